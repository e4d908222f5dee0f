// Two-tile flash attention forward (attention_fwd2_impl.cuh), built for head dimensions 128 and 64.
#include <cstdlib>

#include "common.cuh"
#include "runtime.cuh"

using namespace dd;

#define DD_HEAD_DIM 128
#define DD_FWD2_NS fwd2_d128
#include "attention_fwd2_impl.cuh"
#undef DD_HEAD_DIM
#undef DD_FWD2_NS

#define DD_HEAD_DIM 64
#define DD_FWD2_NS fwd2_d64
#include "attention_fwd2_impl.cuh"
#undef DD_HEAD_DIM
#undef DD_FWD2_NS

// Whether the forward pass should run with two query tiles per CTA.  An odd number of tiles leaves one CTA of a head half
// empty, and with full attention, where every sweep has the same length, few heads finish no later with a tile per SM:
// us, one tile -> two, batch x tokens, heads, full: 1 x 384, 32 of 64: 14.3 -> 16.4; 1 x 640, 8 of 128: 16.4 -> 18.4, of 64:
// 14.4 -> 15.8; but more tiles than SMs 4 x 384, 16 of 64: 24.6 -> 16.4, 1 x 640, 32 of 128: 34.8 -> 22.5, and one tile
// 4 x 128, 16 of 64: 12.2 -> 10.2; causal 1 x 640, 8 of 128: 20.5 -> 18.4.
DD_API int dd_attn_fwd_two_tiles(int batch, int S, int Hq, int causal) {
  if (S % 256 != 128 || causal || S <= 128) return 1;
  return (long long)batch * Hq * (S / 128) > current_sm_count();
}

// softmax(scale * q k^T) v over [batch * S, heads, Dh] bf16 tensors, Dh = 128 or 64, any S: q / k / v by address, row and
// head stride (in elements, unit stride within a row), out contiguous, lse [batch][Hq][S] (may be null).
DD_API int dd_attn_fwd2(const void* q, long long q_row_stride, long long q_head_stride, const void* k,
                        long long k_row_stride, long long k_head_stride, const void* v, long long v_row_stride,
                        long long v_head_stride, void* out, float* lse, int batch, int S, int Hq, int Hkv, int Dh,
                        int causal, float scale, void* stream) {
  if (Dh == 128)
    return fwd2_d128::run(q, q_row_stride, q_head_stride, k, k_row_stride, k_head_stride, v, v_row_stride,
                          v_head_stride, out, lse, batch, S, Hq, Hkv, Dh, causal, scale, stream);
  if (Dh == 64)
    return fwd2_d64::run(q, q_row_stride, q_head_stride, k, k_row_stride, k_head_stride, v, v_row_stride,
                         v_head_stride, out, lse, batch, S, Hq, Hkv, Dh, causal, scale, stream);
  return DD_ERR_BAD_ARG;
}
