// C entry point of the tcgen05 GEMM.
#include <algorithm>
#include <cstdlib>

#include "gemm2_tcgen05.cuh"
#include "gemm4_tcgen05.cuh"
#include <cstring>

#include "gemm_tcgen05.cuh"
#include "runtime.cuh"

using namespace dd;
using namespace dd::gemm;

namespace {
template <bool A_MN, bool B_MN>
int launch(const CUtensorMap& ta, const CUtensorMap& tb, const Params& p, const Plan& plan, int ctas, bool ahead,
           cudaStream_t stream) {
  const int grid = plan.items < ctas ? plan.items : ctas;
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  auto kern = gemm_bf16_kernel<A_MN, B_MN>;
  if (!configured[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e != cudaSuccess) return (int)e;
    configured[dev & 63] = true;
  }
  return launch_ahead(kern, grid, NUM_THREADS, SMEM_BYTES, stream, ahead, ta, tb, p, plan);
}
template <bool A_MN, bool B_MN, int NB>
int launch_pair(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const Params& p, int pairs,
                const dd::gemm2::Plan& plan, cudaStream_t stream) {
  const int grid = 2 * (plan.items < pairs ? plan.items : pairs);
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  auto kern = dd::gemm2::gemm2_bf16_kernel<A_MN, B_MN, NB>;
  constexpr int bytes = dd::gemm2::Shape<NB>::SMEM;
  if (!configured[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return (int)e;
    configured[dev & 63] = true;
  }
  return launch_ahead(kern, grid, dd::gemm2::NUM_THREADS, bytes, stream, !(p.flags & F_ALONE), ta, tb, td, p, plan);
}

template <bool A_MN, bool B_MN>
int launch_wide(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& td, const Params& p,
                const dd::gemm4::Plan& plan, int grid, cudaStream_t stream) {
  static bool configured[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  auto kern = dd::gemm4::gemm4_bf16_kernel<A_MN, B_MN>;
  if (!configured[dev & 63]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, dd::gemm4::SMEM);
    if (e != cudaSuccess) return (int)e;
    configured[dev & 63] = true;
  }
  return launch_ahead(kern, grid, dd::gemm4::NUM_THREADS, dd::gemm4::SMEM, stream, !(p.flags & F_ALONE), ta, tb, td, p,
                      plan);
}

// Second half of a split contraction: D (+)= sum_s part[s] (+ bias), the parts in order (the same bits in every
// run).  Bound by the read of the parts, which the GEMM has just left in L2; four columns per thread.
__global__ void __launch_bounds__(256)
split_reduce_kernel(const float* part, int split, long long part_stride, int ldw, const Params p) {
  const int quads = ldw >> 2;
  const long long total = (long long)p.M * quads;
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  grid_dependency_wait();
  if (i >= total) return;
  const int row = (int)(i / quads), col = (int)(i - (long long)row * quads) * 4;
  const float* src = part + (long long)row * ldw + col;
  float4 s = *reinterpret_cast<const float4*>(src);
#pragma unroll 4
  for (int k = 1; k < split; ++k) {
    const float4 t = *reinterpret_cast<const float4*>(src + k * part_stride);
    s.x += t.x; s.y += t.y; s.z += t.z; s.w += t.w;
  }
  float v[4] = {s.x, s.y, s.z, s.w};
  const bool add = (p.flags & F_ACCUMULATE) != 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    if (col + j >= p.N) break;
    if (p.flags & F_BIAS)
      v[j] += (p.flags & F_BIAS_F32) ? reinterpret_cast<const float*>(p.bias)[col + j]
                                     : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p.bias)[col + j]);
  }
  const long long at = (long long)row * p.ldd + col;
  const bool vec = col + 4 <= p.N && p.ldd % 4 == 0 && (reinterpret_cast<uintptr_t>(p.D) & 15) == 0;
  if (p.flags & F_OUT_F32) {
    float* d = reinterpret_cast<float*>(p.D) + at;
    if (vec) {
      const float4 o = add ? *reinterpret_cast<const float4*>(d) : make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float4*>(d) = make_float4(v[0] + o.x, v[1] + o.y, v[2] + o.z, v[3] + o.w);
    } else {
      for (int j = 0; j < 4 && col + j < p.N; ++j) d[j] = add ? d[j] + v[j] : v[j];
    }
  } else {
    __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(p.D) + at;
    if (vec && !add) {
      *reinterpret_cast<uint2*>(d) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
    } else {
      for (int j = 0; j < 4 && col + j < p.N; ++j)
        d[j] = __float2bfloat16(add ? __bfloat162float(d[j]) + v[j] : v[j]);
    }
  }
}

// Columns of a pair's tile: 128 where the waves of half tiles are the shorter time.  A half tile costs 1.25 times as
// much per column (its operands and what TMA brings are 192 bytes of shared memory a clock, a whole one's are 128).
// Forward, in us, 256 -> 128 columns: 4096 x 1600 x 6400 74.8 -> 69.7, 512 x 1024 x 512 14.3 -> 11.2; 3000 x 2048 x 5632, whose
// last wave of whole tiles is short enough to be taken in halves, 59 -> 63.5; but 4096 x 6400 x 1600 62.4 -> 71.7, 3000 x 11264 x 2048 98 -> 114.  Gradients that are added in fp32
// are bound by their epilogue besides (3000 x 2048 x 5632 70.6 -> 79.9): only where there is one wave either way.
long long whole_tile_waves(long long tiles, long long pairs) {      // in 200ths
  const long long rest = tiles % pairs;                       // (a last, short wave of whole tiles is taken in halves)
  return tiles / pairs * 200 + (rest == 0 ? 0 : tiles > pairs && rest * 2 <= pairs ? 125 : 200);
}
bool half_tiles(int M, int N, int batch, bool f32, long long pairs, long long* whole, long long* half) {
  const long long rows_of_tiles = (long long)((M + 2 * gemm2::BM - 1) / (2 * gemm2::BM)) * batch;
  *whole = rows_of_tiles * ((N + 255) / 256);
  *half = rows_of_tiles * ((N + 127) / 128);
  return f32 ? *half <= pairs : (*half + pairs - 1) / pairs * 125 < whole_tile_waves(*whole, pairs);
}

// Order of a pair kernel's tiles of 256 x 256 (see tile_coords).  Large products run at the power limit, where each byte
// that is read again from memory costs clock: a panel of the operand with fewer rows is kept in L2 (up to 36 MB of it; 67
// MB no longer stay) while the other one streams past it, but at least 8 tiles wide, so that the tiles in flight are about
// square.  In us, back to back, 4 rows before -> now: 8192 x 28672 x 4096 1634 -> 1425 (8 rows 1527), 4096 x 50304 x 1600
// 570 -> 517, 3000 x 32000 x 2048 341 -> 311; 8192 x 4096 x 28672 1619 -> 1511 by columns (8 rows 1529).  A contraction of up to
// 512 moves more of D than of its operands, which stay in L2 anyway, and memory takes whole rows of D sooner than strips of them:
// four rows of tiles, 7582 x 9272 x 64 bf16 57 -> 62 us with a panel of thirty, x 256 60 -> 66, x 512 added in fp32 137 -> 143, but x
// 1024 112 -> 106.
int tile_group(int M, int N, int K) {
  if (K <= 512) return 4;
  const int tiles = (min(M, N) + 255) / 256;
  const int g = min(tiles, max(8, (int)(36000000ll / (512ll * K))));
  return M <= N ? g : -g;
}

// Whether entries with live rows take tiles of 512 x 256.  Only that kernel deals the live blocks out evenly, but at a coarser
// grain and, tile for tile, some 5 % slower where both are even.  The counts are on the device: it is reckoned with four fifths
// of the rows live, what a capacity of 1.25 leaves on average.  With an even number of row blocks the others' tiles lie on every
// other pair, so that pairs with a dead block in each period wait for those without; there from 12 waves or 3e11 operations on.
// Products of 1e12 run at the power limit, where the bytes that wide tiles leave out count (8 x 1280, 990 to 1055 rows live, 28672 x
// 4096, 4096 x 14336, 14336 x 4096, 4096 x 28672: 1754 -> 1666, 959 -> 860, 945 -> 838, 1761 -> 1509 us).  Contractions of up
// to 512 are bound by what is stored, which this kernel does in two sets of warps.  1142 products of 4 to 16 entries of 257 to
// 3000 rows, time against 256-row tiles in groups of four rows: capacities filled to 0.8 0.92, at random 0.93, to 0.03 0.92, full
// 0.94; with the wide tiles in all of them 0.98, 0.95, 0.99, 1.04, and up to 2.1 for one; back to back for half a second, 245
// products from 5e10 operations on, 0.97 and, with the wide tiles in all, 1.00, up to 1.56.  Four fifths of 320 rows are one block,
// but of 8 entries with 246 to 266 live rows half have two, 4096 x 14336 327 -> 406 us: the wide tiles are reckoned with half of
// the last block on average.
bool live_rows_wide(int M, int N, int K, int batch, long long pairs) {
  const long long blocks = (M + 255) / 256, cols = (N + 255) / 256;
  const long long live = std::min(blocks, (M * 4ll + 5 * 256 - 1) / (5 * 256));
  const long long longest = blocks % 2 == 0 && live < blocks ? (live + 1) / 2 * 2 : live;      // live blocks as if all pairs had the most
  const long long tiles = batch * longest * cols;
  if (K <= 512) return tiles >= 4 * pairs;
  const double flops = 2.0 * batch * M * N * K;
  if (live == blocks || flops >= 1e12) return live < blocks;
  const long long mean = std::min(blocks * 1280, M * 4ll + 640);       // live blocks of an entry, in parts of 1280
  const long long slots = (batch * cols * mean + 2 * 1280 - 1) / (2 * 1280);
  const long long waves = (tiles + pairs - 1) / pairs, wide = (slots + pairs - 1) / pairs * 2;
  return (tiles >= 12 * pairs || flops >= 3e11) && wide * 100 < waves * 95;
}

// Which kernel takes a product, with how many CTAs, its work items and the order of its tiles.
enum Kernel : int { SINGLE, PAIR, PAIR_HALF, WIDE };
struct Choice {
  Kernel kernel;
  int ctas, group_m;
  bool ahead;                        // launched ahead of the end of the kernel before it
  Plan single;                       // (of the kernel that is taken; the others are not set)
  dd::gemm2::Plan pair;
  dd::gemm4::Plan wide;
};

// flags with F_TMA_EPI where the output allows it; rows: A has live rows or, with bound_k, live terms; a_span: bytes from the first
// element of A to behind its last.
Choice choose(int M, int N, int K, int batch, int flags, int max_ctas, bool rows, bool bound_k, long long a_span) {
  Choice c = {};
  const int sms = current_sm_count();
  c.ahead = !(max_ctas > 0 && max_ctas < sms);
  // CTA pairs (cta_group::2) unless disabled or the problem is a single tile row
  static const bool pair_ok = []() { const char* e = getenv("DISTDL_GEMM_PAIR"); return !(e && e[0] == '0'); }();
  if (!pair_ok || M <= BM) {
    c.kernel = SINGLE;
    c.ctas = max_ctas > 0 && max_ctas < sms ? max_ctas : sms;
    c.group_m = 8;
    c.single = make_plan(M, N, batch, c.ctas, a_span);
    // Many CTAs on an A that lies close together are slower on SMs that the product before leaves idle (they wait for one
    // another's reads, see make_plan, more so the more uneven they lie).  Products of different weights in a chain, us, not ahead
    // -> ahead: 1 x 14336 x 4096 (56 items) 36 -> 42, 8 x 24576 x 4096 49 -> 54, 1 x 50176 x 8192 162 -> 167; 1 x 12288 x 1024 (48 items)
    // 12.5 -> 11.3, 33 x 14336 x 4096 (no such A) 29.5 -> 28.6.
    if (a_span < kNearA && c.single.items > 48) c.ahead = false;
    return c;
  }
  c.ctas = sms & ~1;
  if (max_ctas > 0 && max_ctas < c.ctas) c.ctas = max_ctas & ~1;
  if (c.ctas < 2) c.ctas = 2;
  const int pairs = c.ctas / 2;
  long long whole, half;
  const bool narrow = half_tiles(M, N, batch, (flags & F_OUT_F32) != 0, pairs, &whole, &half) && !rows;
  // Tiles of 512 x 256 (gemm4_tcgen05.cuh) for at least a whole wave of them.  They bring a quarter less through L2, but
  // pairs wait for the epilogue between tiles, and the order of tiles that keeps a panel in L2 is at its best with the
  // smaller ones where the contraction is short.  In us, back to back, 256 rows -> 512 rows: K = 1600: 4096 x 50304
  // 515 -> 531; K = 4096: 8192 x 28672 1441 -> 1448; K = 8192: 8192 x 8192 895 -> 842, weight gradient 28672 x 4096
  // 1649 -> 1533; K = 14336: 8192 x 4096 768 -> 741; K = 128256: 8192 x 4096 7756 -> 6838.
  // Where their waves end later than those of the smaller tiles by more than the traffic gains, these stay: weight gradient
  // 5184 x 1728 of 7716 rows, 147 tiles in two waves, or 77 in one of twice the length and one more; a training step that has it
  // 8 680 -> 8 440 us, 9 030 with the larger tiles there.
  // Entries with live rows: live_rows_wide.
  const bool by_rows = rows && !bound_k && live_rows_wide(M, N, K, batch, pairs);
  if (!narrow && (flags & F_TMA_EPI) && (by_rows || (!rows && K > 4096)) && M > 256) {
    c.wide = dd::gemm4::make_plan(M, N, batch, pairs);
    const long long waves = (long long)(c.wide.full + pairs - 1) / pairs * 400 + (c.wide.items > c.wide.full ? 200 : 0);
    if (c.wide.full > 0 && (by_rows || waves * 100 <= whole_tile_waves(whole, pairs) * 106)) {
      c.kernel = WIDE;
      c.group_m = M <= N ? 8 : -16;
      return c;
    }
  }
  c.kernel = narrow ? PAIR_HALF : PAIR;
  // (four rows of half tiles: 4096 x 1600 x 6400 76 us, 79 to 83 in the other orders; and by columns, tiles without live rows
  // follow one another on the same pairs: 16 x 1698 x 576 x 10496, 7 to 81 rows live, 72 us by rows, 150 by columns)
  c.group_m = narrow || (rows && !bound_k && M > N) ? 4 : tile_group(M, N, K);
  c.pair = dd::gemm2::make_plan(M, N, batch, pairs, narrow ? 128 : 256);
  return c;
}
}  // namespace

// D[b,m,n] (+)= sum_k A[b,m,k] B[b,n,k] (+ bias[n]);  bf16 operands, fp32 accumulation.
//   a_mn / b_mn : 0 = K-major (lda = elements between rows m / n),
//                 1 = MN-major (lda = elements between rows k)
//   stride*     : elements between batches (ignored when batch == 1)
//   flags       : dd::gemm::Flags
//   max_ctas    : 0 = one CTA per SM; otherwise an upper bound, which leaves
//                 SMs to a concurrent communication kernel: until the product
//                 has ended, the kernel behind it does not start on them either
namespace {
int gemm_bf16(const void* A, int a_mn, long long lda, long long strideA, const void* B, int b_mn, long long ldb,
              long long strideB, void* D, long long ldd, long long strideD, const void* bias, int M, int N, int K,
              int batch, int flags, int max_ctas, const int* rows, int bound_k, void* stream, bool parts_of_k = false) {
  if (M <= 0 || N <= 0 || K <= 0 || batch <= 0) return DD_ERR_BAD_ARG;
  if ((lda % 8) || (ldb % 8)) return DD_ERR_ALIGN;
  if (batch > 1 && ((strideA % 8) || (strideB % 8))) return DD_ERR_ALIGN;
  if (batch == 1) {
    strideA = (a_mn ? (long long)K : (long long)M) * lda;
    strideB = (b_mn ? (long long)K : (long long)N) * ldb;
    strideD = (long long)M * ldd;
  }
  if (max_ctas > 0 && max_ctas < current_sm_count()) flags |= F_ALONE;
  // TMA epilogue of the pair kernels where the output qualifies: bf16 store, fp32 store or fp32 add
  static const bool tma_epi = []() { const char* e = getenv("DISTDL_GEMM_TMA_EPI"); return !(e && e[0] == '0'); }();
  const bool f32 = (flags & F_OUT_F32) != 0;
  const long long es = f32 ? 4 : 2;
  const bool tma_out = tma_epi && (f32 || !(flags & F_ACCUMULATE)) && (reinterpret_cast<uintptr_t>(D) & 15) == 0 &&
                       (ldd * es) % 16 == 0 && (strideD * es) % 16 == 0;
  // (parts of one contraction: each reads a part of A of its own, and briefly)
  const long long a_span = parts_of_k ? 1ll << 62 : 2 * ((batch - 1) * strideA + (a_mn ? (K - 1) * lda + M : (M - 1) * lda + K));
  const Choice c = choose(M, N, K, batch, flags | (tma_out ? F_TMA_EPI : 0), max_ctas, rows != nullptr, bound_k != 0, a_span);
  int err = 0, r;
  Params p;
  p.M = M; p.N = N; p.K = K; p.batch = batch;
  p.D = D; p.ldd = ldd; p.strideD = strideD; p.bias = bias; p.flags = flags; p.group_m = c.group_m;
  p.status = device_status(&err);
  if (err) return err;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  CUtensorMap ta, tb, td;
  static_assert(BM == dd::gemm2::BM && BK == dd::gemm2::BK && BM == dd::gemm4::BLK / 2 && BK == dd::gemm4::BK, "boxes of A");
  if (a_mn) r = get_tensor_map_bf16_3d(&ta, A, M, K, batch, lda * 2, strideA * 2, 64, BK);
  else      r = get_tensor_map_bf16_3d(&ta, A, K, M, batch, lda * 2, strideA * 2, BK, BM);
  if (r) return r;
  if (b_mn) r = get_tensor_map_bf16_3d(&tb, B, N, K, batch, ldb * 2, strideB * 2, 64, BK);
  else      r = get_tensor_map_bf16_3d(&tb, B, K, N, batch, ldb * 2, strideB * 2, BK, 64);
  if (r) return r;
  if (c.kernel == SINGLE) {
    if (a_mn && b_mn) return launch<true, true>(ta, tb, p, c.single, c.ctas, c.ahead, s);
    if (a_mn) return launch<true, false>(ta, tb, p, c.single, c.ctas, c.ahead, s);
    if (b_mn) return launch<false, true>(ta, tb, p, c.single, c.ctas, c.ahead, s);
    return launch<false, false>(ta, tb, p, c.single, c.ctas, c.ahead, s);
  }
  p.rows = rows; p.bound_k = bound_k;
  memset(&td, 0, sizeof(td));
  if (tma_out) {
    r = f32 ? get_tensor_map_f32_3d(&td, D, N, M, batch, ldd * 4, strideD * 4, 32, 32)
            : get_tensor_map_bf16_3d(&td, D, N, M, batch, ldd * 2, strideD * 2, 64, 32);
    if (r) return r;
    p.flags |= F_TMA_EPI;
  }
  const int pairs = c.ctas / 2;
  if (c.kernel == WIDE) {
    const int grid = 2 * (c.wide.items < pairs ? c.wide.items : pairs);
    if (a_mn && b_mn) return launch_wide<true, true>(ta, tb, td, p, c.wide, grid, s);
    if (a_mn) return launch_wide<true, false>(ta, tb, td, p, c.wide, grid, s);
    if (b_mn) return launch_wide<false, true>(ta, tb, td, p, c.wide, grid, s);
    return launch_wide<false, false>(ta, tb, td, p, c.wide, grid, s);
  }
  if (c.kernel == PAIR_HALF) {
    if (a_mn && b_mn) return launch_pair<true, true, 128>(ta, tb, td, p, pairs, c.pair, s);
    if (a_mn) return launch_pair<true, false, 128>(ta, tb, td, p, pairs, c.pair, s);
    if (b_mn) return launch_pair<false, true, 128>(ta, tb, td, p, pairs, c.pair, s);
    return launch_pair<false, false, 128>(ta, tb, td, p, pairs, c.pair, s);
  }
  if (a_mn && b_mn) return launch_pair<true, true, 256>(ta, tb, td, p, pairs, c.pair, s);
  if (a_mn) return launch_pair<true, false, 256>(ta, tb, td, p, pairs, c.pair, s);
  if (b_mn) return launch_pair<false, true, 256>(ta, tb, td, p, pairs, c.pair, s);
  return launch_pair<false, false, 256>(ta, tb, td, p, pairs, c.pair, s);
}
}  // namespace

DD_API int dd_gemm_bf16(const void* A, int a_mn, long long lda, long long strideA, const void* B, int b_mn,
                        long long ldb, long long strideB, void* D, long long ldd, long long strideD,
                        const void* bias, int M, int N, int K, int batch, int flags, int max_ctas,
                        void* stream) {
  return gemm_bf16(A, a_mn, lda, strideA, B, b_mn, ldb, strideB, D, ldd, strideD, bias, M, N, K, batch, flags, max_ctas,
                   nullptr, 0, stream);
}

// The same for a batch whose entry b has zeros in A after its first rows[b] rows (bound_k: whose terms of the
// contraction after the first rows[b] are zero); rows [batch] on the device.  The result is the same: what is known
// to be zero is not read and not multiplied, in tiles of 256 rows or blocks of 64 terms (by the CTA-pair kernel).
DD_API int dd_gemm_bf16_rows(const void* A, int a_mn, long long lda, long long strideA, const void* B, int b_mn,
                             long long ldb, long long strideB, void* D, long long ldd, long long strideD, int M, int N,
                             int K, int batch, int flags, const int* rows, int bound_k, void* stream) {
  return gemm_bf16(A, a_mn, lda, strideA, B, b_mn, ldb, strideB, D, ldd, strideD, nullptr, M, N, K, batch, flags, 0, rows,
                   bound_k, stream);
}

// What the entries above would do with a contiguous A and an output that TMA can write, for tests: the kernel (0 single CTA, 1
// pair, 2 pair with half tiles, 3 512 x 256 per pair), CTAs at most, order of tiles, whole tiles, work items, parts of a tile
// behind the whole ones, and whether it is launched ahead.
DD_API int dd_gemm_plan(int M, int N, int K, int batch, int flags, int max_ctas, int rows, int bound_k, int* out) {
  if (M <= 0 || N <= 0 || K <= 0 || batch <= 0) return DD_ERR_BAD_ARG;
  const Choice c = choose(M, N, K, batch, flags | F_TMA_EPI, max_ctas, rows != 0, bound_k != 0, 2ll * batch * M * K);
  out[0] = c.kernel; out[1] = c.ctas; out[2] = c.group_m;
  out[3] = c.kernel == SINGLE ? c.single.full : c.kernel == WIDE ? c.wide.full : c.pair.full;
  out[4] = c.kernel == SINGLE ? c.single.items : c.kernel == WIDE ? c.wide.items : c.pair.items;
  out[5] = c.kernel == SINGLE ? c.single.parts : 2;
  out[6] = c.ahead;
  return DD_OK;
}

// Into how many parts dd_gemm_bf16_split should cut the contraction (1: not at all).  A GEMM with few output tiles
// leaves SMs idle while each of its own walks all of K, and an SM takes in no more than about 85 GB/s, so that even
// the read of the weights goes at a fifth of the memory rate with 16 tiles.  The parts run as a batch of the same
// kernels into an fp32 workspace.  Measured, each alone and with a cold L2: 33 x 4096 x 14336 split 8 ways 79 -> 40 us,
// 33 x 64 x 4096 16 ways 25.6 -> 13.3, 200 x 2048 x 8192 8 ways 33.7 -> 27.6, error against fp64 2 to 10 times smaller (shorter
// sums).  A k-block of 64 costs a CTA about 0.36 us, the parts and their sum about 5 us, the second launch 8 us on the host,
// which a short GEMM does not hide: split from a gain of 8 us beyond both on.  That is reckoned for whole tiles; up to 128 rows
// halves of tiles cost 0.34 and quarters 0.29, so that the device gains less there than the rule says: 8 us or more at 150 of 164
// sizes of 33 and 128 rows that are split, 3 to 8 at most others (128 x 6144 x 6144 6 ways 43.2 -> 39.9), nothing at 128 x 14336
// x 11264.  A k-block of half tiles costs a pair 0.20 us:
// nothing is split whose parts gain nothing over the product that takes them (1000 x 2048 x 14336, parts of whole tiles:
// 55.3 us, 2 ways 58.3; 512 x 4096 x 11264 51.2, 2 ways 54.2).
DD_API int dd_gemm_split(int M, int N, int K) {
  const int sms = current_sm_count(), num_k = K / 64;
  if (K % 64 || M <= 0 || N <= 0) return 1;
  const bool pair = M > BM;
  const long long tiles = (long long)((M + (pair ? 2 * BM - 1 : BM - 1)) / (pair ? 2 * BM : BM)) * ((N + BN - 1) / BN);
  const long long slots = pair ? sms / 2 : sms;
  long long whole, half;
  const double block = pair && half_tiles(M, N, 1, false, slots, &whole, &half) ? 0.20 : 0.36;
  int best = 1;
  double best_gain = 8.0;
  for (int s = 2; s <= 16 && tiles * s <= slots && num_k / s >= 4; ++s) {
    if (num_k % s) continue;
    const double sum = 5.0 + (double)s * M * N * 8.0 / 6e6, gain = 0.36 * (num_k - num_k / s) - 8.0 - sum;
    const double part = pair && half_tiles(M, N, s, true, slots, &whole, &half) ? 0.20 : 0.36;
    if (block * num_k - part * (num_k / s) < sum) continue;
    if (gain > best_gain) { best_gain = gain; best = s; }
  }
  return best;
}

// dd_gemm_bf16 for one product whose contraction runs in `split` parts (K a multiple of 64 * split).
// ws: split * M * (N rounded up to 4) floats, 16-byte aligned.
DD_API int dd_gemm_bf16_split(const void* A, int a_mn, long long lda, const void* B, int b_mn, long long ldb, void* D,
                              long long ldd, const void* bias, int M, int N, int K, int flags, int split, float* ws,
                              void* stream) {
  if (M <= 0 || N <= 0 || split < 1 || K <= 0 || K % (64 * split) || ws == nullptr) return DD_ERR_BAD_ARG;
  if (reinterpret_cast<uintptr_t>(ws) & 15) return DD_ERR_ALIGN;
  const long long kc = K / split;
  const int ldw = (N + 3) & ~3;
  const int r = gemm_bf16(A, a_mn, lda, a_mn ? kc * lda : kc, B, b_mn, ldb, b_mn ? kc * ldb : kc, ws, ldw,
                          (long long)M * ldw, nullptr, M, N, (int)kc, split, F_OUT_F32, 0, nullptr, 0, stream, true);
  if (r) return r;
  Params p;
  p.M = M; p.N = N; p.K = K; p.batch = 1;
  p.D = D; p.ldd = ldd; p.strideD = 0; p.bias = bias; p.flags = flags; p.group_m = 1; p.status = nullptr;
  const long long total = (long long)M * (ldw / 4);
  return launch_ahead(split_reduce_kernel, (unsigned)((total + 255) / 256), 256, 0, reinterpret_cast<cudaStream_t>(stream),
                      true, ws, split, (long long)M * ldw, ldw, p);
}
