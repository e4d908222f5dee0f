// Flash attention backward (attention_bwd3_impl.cuh), built for head dimensions 128 and 64.
#include <cstdlib>

#include "common.cuh"
#include "runtime.cuh"

using namespace dd;

namespace dd {
// Grouped-query heads: one CTA per key tile and kv head sweeps the heads of the group one after the other (their
// queries and sums of dQ then stay in L2, one head of a group at a time), or, where the longest sweep would be longer
// than an SM's share of all tile pairs, one per query head, which add their dV and dK in the order of the heads.
int bwd3_split(int batch, int nT, int Hq, int Hkv, int causal) {
  const long long kv_heads = (long long)batch * Hkv, sweeps = causal ? kv_heads * (nT + 1) / 2 : kv_heads * nT;
  return Hq > Hkv && sweeps < current_sm_count() ? Hq / Hkv : 1;
}
// Words of scratch: per 128 queries of a head two statistics each and two counters; with more than one key tile the sums of
// dQ, with the heads of a group split those of dK and dV.
long long bwd3_words(int batch, int S, int Hq, int Hkv, int Dh, int causal) {
  const int nT = S / 128 + (S % 128 != 0);
  const long long tiles = (long long)batch * Hq * nT, kv_tiles = (long long)batch * Hkv * nT;
  return 256 * tiles + 4 + (2 * tiles + 3) / 4 * 4 + (nT > 1 ? 128 * Dh * tiles : 0) +
         (bwd3_split(batch, nT, Hq, Hkv, causal) > 1 ? 256 * Dh * kv_tiles : 0);
}
}  // namespace dd

#define DD_HEAD_DIM 128
#define DD_BWD3_NS bwd3_d128
#include "attention_bwd3_impl.cuh"
#undef DD_HEAD_DIM
#undef DD_BWD3_NS

#define DD_HEAD_DIM 64
#define DD_BWD3_NS bwd3_d64
#include "attention_bwd3_impl.cuh"
#undef DD_HEAD_DIM
#undef DD_BWD3_NS

// Gradients of softmax(scale * q k^T) v over [batch * S, heads, Dh] bf16 tensors given by address, row and head stride;
// out and dout are contiguous, lse is [batch][Hq][S].  `scratch` holds `words` words, no fewer than dd_attn_bwd_one_pass says.
DD_API int dd_attn_bwd3(const void* q, long long q_row, long long q_head, const void* k, long long k_row,
                       long long k_head, const void* v, long long v_row, long long v_head, const void* out,
                       const void* dout, const float* lse, float* scratch, long long words, void* dq, long long dq_row,
                       long long dq_head, void* dk, long long dk_row, long long dk_head, void* dv, long long dv_row,
                       long long dv_head, int batch, int S, int Hq, int Hkv, int Dh, int causal, float scale,
                       void* stream) {
  auto run = Dh == 128 ? bwd3_d128::run : Dh == 64 ? bwd3_d64::run : nullptr;
  if (run == nullptr) return DD_ERR_BAD_ARG;
  return run(q, q_row, q_head, k, k_row, k_head, v, v_row, v_head, out, dout, lse, scratch, words, dq, dq_row, dq_head, dk,
             dk_row, dk_head, dv, dv_row, dv_head, batch, S, Hq, Hkv, causal, scale, stream);
}

// Whether a backward pass should run in one kernel (attention_bwd3_impl.cuh) or in two (attention_bwd2_impl.cuh, whole
// tiles only).  The one kernel forms the scores once and one exponential per score, but its CTAs hand the sums of dQ on to
// one another (the key tiles of a head that start together follow one another at a distance of 3 us, and a delay of
// one is a delay of all behind it), and at head dim 128 shared memory bounds it at nearly the time of the two.  In us, two
// kernels -> one, batch x tokens, heads:
//   head dim 64    8 x 1536, 16: 577 -> 392    4 x 1024, 25, causal: 173 -> 128    16 x 512, 16: 169 -> 149
//                  1 x 16384, 16: 4963 -> 3486    1 x 4096, 8, causal, 18 of 32 key tiles together: 119 -> 136
//   head dim 128   heads of a group split: 3 x 1024, 16 / 4, causal: 149 -> 112; 1 x 16384, 4 / 1, causal: 1379 -> 906
//                  one key tile: 64 x 128, 16 / 4: 118 -> 75    1 x 16384, 32 / 8, causal: 6667 -> 6109
//                  8 x 1024, 32, causal: 464 -> 507    2 x 2048, 16: 276 -> 314    2 x 4096, 32 / 8, causal: 1050 -> 1058
// Hence: always where the group's heads are split over CTAs (the two kernels leave SMs idle there) and for one key tile;
// otherwise where no more than a quarter of a head's key tiles start together, at head dim 128 for long sweeps only.
// `words`: of scratch for the one kernel, on this device.
DD_API int dd_attn_bwd_one_pass(int batch, int S, int Hq, int Hkv, int Dh, int causal, long long* words) {
  *words = 4;
  if (S <= 0 || batch <= 0 || Hkv <= 0 || Hq <= 0) return 1;         // (refused by the kernel's entry)
  *words = dd::bwd3_words(batch, S, Hq, Hkv, Dh, causal);
  if (S % 128) return 1;
  const int nT = S / 128;
  if (nT <= 1 || dd::bwd3_split(batch, nT, Hq, Hkv, causal) > 1) return 1;
  const long long fit = current_sm_count() / ((long long)Hkv * batch);
  const long long together = fit < 1 ? 1 : fit < nT ? fit : nT;
  return (together == 1 || together * 4 <= nT) && (Dh == 64 || nT >= 64);
}
