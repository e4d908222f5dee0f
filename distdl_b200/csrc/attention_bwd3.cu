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

// Whether the backward pass of a group that is split over CTAs is faster in one kernel than in two.  What the two kernels
// leave idle shrinks with the pairs of kv head and key tile (`kv_tiles`), since they have one CTA for each; what the one
// kernel loses is the hand-over.  Ratios one kernel : two, cold L2, by kv_tiles (800 sizes measured in all):
//   head dim 128, causal   2 tiles, groups of 4:  48 0.82  112 1.03  176 1.17    2 tiles, groups of 8:  48 1.02  112 1.17
//                          8 tiles, groups of 4:  80 0.76  144 0.94  208 1.16   16 tiles, groups of 8: 112 0.77  176 1.03
//                         48 tiles, groups of 8: 144 0.69  240 0.94             32 tiles, groups of 2: 192 0.89  256 1.11
//   head dim 128, full     groups of 4: 2 tiles 32 0.96 64 1.11, 8 tiles 32 1.19, 32 tiles 96 1.27
//                          groups of 8: 4 tiles 32 0.96 64 1.06, 16 tiles 64 0.90 96 1.15
//   head dim 64, full      groups of 2: 2 tiles 32 0.94 64 1.06, 8 tiles 32 1.29    groups of 3: 4 tiles 32 0.95, 24 tiles 24 1.12
//                          groups of 4: 2 tiles 100 1.09, 16 tiles 96 0.89          (causal: 0.37 to 1.00)
static bool split_in_one_pass(int nT, int group, long long kv_tiles, int Dh, int causal, long long sms) {
  if (Dh == 64) {
    if (causal) return true;
    if (nT <= 4 && (nT <= 2 ? kv_tiles * 2 > sms : kv_tiles * 3 > sms * 2)) return false;
    return group > 3 || nT <= (group == 3 ? 8 : 2);
  }
  if (causal) return kv_tiles * 5 * (nT + group) <= 8 * sms * nT || nT >= 64;
  if (group >= 6 && nT * 4 >= group) return nT >= 8 ? kv_tiles * 5 <= sms * 2 : kv_tiles * 3 <= sms;
  return (nT <= 2 || group == 5) && nT * 4 >= group && kv_tiles * 4 <= sms;
}

// Whether a backward pass should run in one kernel (attention_bwd3_impl.cuh) or in two (attention_bwd2_impl.cuh, whole
// tiles only).  The one kernel forms the scores once and one exponential per score, but its CTAs hand the sums of dQ on to
// one another: the key tiles of a head that start together follow one another at the distance of a hand-over, which
// full attention waits for (every sweep has the same length and starts at the same query tile) and causal attention
// hides behind its longer sweeps.  At head dim 128 shared memory bounds it at nearly the time of the two besides.  Groups
// that are split: above.  Otherwise, in us, two kernels -> one, batch x tokens, heads, each call alone and with a cold L2
// (in brackets: back to back, where the power limit counts and with it the fewer products):
//   head dim 64            8 x 1536, 16: 577 -> 392; 16 x 512, 16: 169 -> 149; 1 x 16384, 16: 5479 -> 3722; but 1 x 4096, 8, causal,
//                          18 of 32 key tiles together: 112 -> 120; 1 x 1024, 16, full, all 8 together: 46 -> 77
//   head dim 128, causal   1 x 16384, 32: 7412 -> 6791 (7581 -> 6679); 1 x 8192, 16: 873 -> 837 (965 -> 886); 1 x 16384, 32 / 8:
//                          6170 -> 6632 (6988 -> 6403); but 8 x 1024, 32: 464 -> 503, 1 x 2048, 16: 93 -> 102
//   head dim 128, full     1 x 16384, 32: 16190 -> 13422 (16588 -> 13371); but 1 x 4096, 8: 261 -> 489; 1 x 16384, 8: 3113 -> 4063;
//                          1 x 16384, 32 / 8: 13976 -> 14919 (13897 -> 14790)
//   one key tile           64 x 128, 16 / 4 of 128: 118 -> 75
// (The two at head dim 128 take 5 % less since their softmax threads work on two values per instruction: 2 x 4096, 32 / 8, causal
// 973 -> 922 back to back.  Measured again, one batch, 485 sizes that take the one kernel: 0.80 of the time of the two on average,
// cold; 26 are slower by 3 to 12 %, most of them groups over two key tiles in full attention, 256 tokens, 48 / 16 of 128 39.9 -> 40.2,
// 192 / 24 81 -> 91, and 8192 tokens, 8 / 4 of 128, causal 400 -> 441.)
// Hence one kernel where no more than a quarter of a head's key tiles start together, at head dim 128 for long sweeps only.
// `words`: of scratch for the one kernel, on this device.
DD_API int dd_attn_bwd_one_pass(int batch, int S, int Hq, int Hkv, int Dh, int causal, long long* words) {
  *words = 4;
  if (S <= 0 || batch <= 0 || Hkv <= 0 || Hq <= 0) return 1;         // (refused by the kernel's entry)
  *words = dd::bwd3_words(batch, S, Hq, Hkv, Dh, causal);
  if (S % 128) return 1;
  const int nT = S / 128;
  if (nT <= 1) return 1;
  const long long sms = current_sm_count();
  if (dd::bwd3_split(batch, nT, Hq, Hkv, causal) > 1 &&
      split_in_one_pass(nT, Hq / Hkv, (long long)batch * Hkv * nT, Dh, causal, sms))
    return 1;
  const long long fit = sms / ((long long)Hkv * batch);
  const long long together = fit < 1 ? 1 : fit < nT ? fit : nT;
  if (Dh == 64) return together == 1 || together * 4 <= nT;
  return nT >= 64 && (causal ? together * 4 <= nT : Hq == Hkv && together * 32 <= nT);
}

// Whether training on a packed projection of a length that is not whole tiles (head dim 128) is faster on the kernels here
// than on the library's operators, which put the packed gradient together by copies but whose backward pass waits for no
// hand-over.  Forward and backward in us, library -> here, batch x tokens, heads:
//   causal   1 x 900, 8: 183 -> 102; 3 x 1000, 32: 411 -> 224; 4 x 3000, 32 / 8: 1660 -> 1456; 1 x 4000, 32 / 8: 671 -> 605; 1 x 6000,
//            32: 1450 -> 1290; but 1 x 4600, 32 / 8: 812 -> 886, 1 x 9000, 32 / 8: 2495 -> 3008, 1 x 12000, 32: 4512 -> 4803
//   full     1 x 600, 32 / 8: 182 -> 105; 1 x 1000, 16: 197 -> 140; 3 x 1531, 32: 738 -> 657; 2 x 1000, 16 / 4: 323 -> 161;
//            4 x 1000, 16 / 8: 368 -> 262; but 1 x 2100, 16: 279 -> 298, 1 x 4000, 8: 390 -> 528, 4 x 1000, 32 / 8: 448 -> 579,
//            1 x 1300, 32 / 8: 220 -> 255, 2 x 3000, 16 / 4: 640 -> 1445
DD_API int dd_attn_ragged(int batch, int S, int Hq, int Hkv, int causal) {
  if (S <= 0 || batch <= 0 || Hkv <= 0 || Hq < Hkv) return 0;
  const int nT = S / 128 + 1, group = Hq / Hkv;
  if (causal) return nT <= (group == 1 ? 64 : 32);
  if (group == 1) return nT <= 12;
  return (long long)group * nT <= 20 || (nT <= 10 && dd::bwd3_split(batch, nT, Hq, Hkv, 0) > 1);
}
