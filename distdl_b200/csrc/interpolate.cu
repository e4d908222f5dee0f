// Nearest-left ("constant") and multilinear interpolation of sub-tensors in
// GLOBAL coordinates, forward and adjoint, 1-3 spatial dimensions, fp32 / fp64 (CUDA also bf16):
// sm_100a kernels plus an OpenMP CPU implementation in the same library (the
// CPU path is the oracle of the GPU tests and serves CPU tensors).
//
// A worker holds the slab [x_off, x_off + in_local) of a global input of extent
// in_global and produces the slab [y_off, y_off + out_local) of the global
// output; index arithmetic uses the global extents, so the shards of a
// partitioned tensor reproduce the serial result exactly.  Conventions are those
// of torch.nn.functional.interpolate: with align_corners the source coordinate
// of output i is i * (in - 1) / (out - 1); otherwise max(0, (i + 0.5) * s - 0.5)
// with s = 1 / scale_factor (or in / out); nearest takes floor(i * s).
// Counterpart of the reference's CPU-only C++ extension
// (src/distdl/functional/interpolate/src/*.cpp).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "common.cuh"

namespace {

struct InterpGeom {
  int in_local[3], out_local[3], x_off[3], y_off[3], in_global[3], out_global[3];
  double scale[3];      // source step per output index (already inverted)
  int align_corners;
  int linear;
};

template <typename T>
__host__ __device__ inline void source_index(const InterpGeom& g, int d, int o_local, int& i0, int& i1, T& lam) {
  const int og = o_local + g.y_off[d];
  const int n_in = g.in_global[d], n_out = g.out_global[d];
  if (!g.linear) {
    int idx = (int)floor((double)og * g.scale[d]);
    if (idx > n_in - 1) idx = n_in - 1;
    i0 = i1 = idx - g.x_off[d];
    lam = (T)0;
    return;
  }
  double src;
  if (g.align_corners) src = (n_out > 1) ? (double)og * (double)(n_in - 1) / (double)(n_out - 1) : 0.0;
  else {
    src = ((double)og + 0.5) * g.scale[d] - 0.5;
    if (src < 0.0) src = 0.0;
  }
  int lo = (int)floor(src);
  if (lo > n_in - 1) lo = n_in - 1;
  const int hi = lo + 1 < n_in ? lo + 1 : lo;
  double l = src - (double)lo;
  if (l < 0.0) l = 0.0;
  if (l > 1.0) l = 1.0;
  if (hi == lo) l = 0.0;
  i0 = lo - g.x_off[d];
  i1 = hi - g.x_off[d];
  lam = (T)l;
}

// CPU: one output element gathers (forward) or scatters (adjoint) its <= 8 corners.
template <typename T, bool ADJOINT>
inline void process_output(const InterpGeom& g, T* x, T* y, long long bc, int o0, int o1, int o2) {
  int a0[3], a1[3];
  T lam[3];
  source_index<T>(g, 0, o0, a0[0], a1[0], lam[0]);
  source_index<T>(g, 1, o1, a0[1], a1[1], lam[1]);
  source_index<T>(g, 2, o2, a0[2], a1[2], lam[2]);
  const long long in_plane = (long long)g.in_local[0] * g.in_local[1] * g.in_local[2];
  const long long out_plane = (long long)g.out_local[0] * g.out_local[1] * g.out_local[2];
  T* xb = x + bc * in_plane;
  T* yo = y + bc * out_plane + ((long long)o0 * g.out_local[1] + o1) * g.out_local[2] + o2;
  T acc = (T)0;
  const T gy = ADJOINT ? *yo : (T)0;
  for (int c = 0; c < 8; ++c) {
    const int s0 = c & 1, s1 = (c >> 1) & 1, s2 = (c >> 2) & 1;
    const T w = (s0 ? lam[0] : (T)1 - lam[0]) * (s1 ? lam[1] : (T)1 - lam[1]) * (s2 ? lam[2] : (T)1 - lam[2]);
    if (w == (T)0) continue;
    const int i0 = s0 ? a1[0] : a0[0], i1 = s1 ? a1[1] : a0[1], i2 = s2 ? a1[2] : a0[2];
    if (i0 < 0 || i0 >= g.in_local[0] || i1 < 0 || i1 >= g.in_local[1] || i2 < 0 || i2 >= g.in_local[2]) continue;
    T* px = xb + ((long long)i0 * g.in_local[1] + i1) * g.in_local[2] + i2;
    if (ADJOINT) {
      *px += w * gy;
    } else {
      acc += w * *px;
    }
  }
  if (!ADJOINT) *yo = acc;
}

// ---------------------------------------------------------------------------------- GPU kernels
// Both directions move each element once and are meant to run at memory speed, so a thread fixes ONE
// spatial position, takes its source rows, columns and weights (fp64 arithmetic) from a table that the CTA
// fills together, and then walks the batch x channel planes.  [8, 64, 128, 128] -> 256^2 in bf16: forward
// 437 -> 76 us, adjoint 420 -> 65 us; [1, 32, 46^3] -> 69^3 in fp32: 208 -> 50 and 205 -> 82 us (before: one element at a time with fp64 index
// arithmetic and fp32 copies of the tensors around the kernel; the adjoint scattered with atomics).
// The adjoint GATHERS: an input position collects the outputs whose support covers it, which makes it
// deterministic and needs neither a cleared gradient nor atomics.
constexpr int kThreads = 256;

template <typename T> struct Acc { using type = T; };
template <> struct Acc<__nv_bfloat16> { using type = float; };
__device__ __forceinline__ float ld(const float* p) { return __ldg(p); }
__device__ __forceinline__ double ld(const double* p) { return __ldg(p); }
__device__ __forceinline__ float ld(const __nv_bfloat16* p) {
  return __uint_as_float((uint32_t)__ldg(reinterpret_cast<const unsigned short*>(p)) << 16);
}
__device__ __forceinline__ void st(float* p, float v) { *p = v; }
__device__ __forceinline__ void st(double* p, double v) { *p = v; }
__device__ __forceinline__ void st(__nv_bfloat16* p, float v) { *p = __float2bfloat16(v); }
// acc + w v, where a zero weight takes nothing from its operand, not even an infinity or a NaN: in fp32 by a mask
// that is made once (two instructions per term), in fp64 by selection
template <typename A> struct Weight;
template <> struct Weight<float> {
  float w;
  uint32_t mask;
  __device__ __forceinline__ void set(float v) { w = v; mask = v != 0.f ? 0xffffffffu : 0u; }
  __device__ __forceinline__ float add(float acc, float v) const {
    return fmaf(w, __uint_as_float(__float_as_uint(v) & mask), acc);
  }
};
template <> struct Weight<double> {
  double w;
  __device__ __forceinline__ void set(double v) { w = v; }
  __device__ __forceinline__ double add(double acc, double v) const { return w != 0.0 ? acc + w * v : acc; }
};
template <typename A> __device__ __forceinline__ A term(A w, A v) { return w != (A)0 ? w * v : (A)0; }

// Where the positions of one CTA lie: consecutive positions of a plane, so that a CTA meets few different
// columns, rows and sheets, and their source indices and weights go into a table in shared memory that the
// CTA's threads fill together (fp64 arithmetic for tens of entries instead of three per thread).
struct Span {
  int col0, row0, sheet0;      // of the CTA's first position
  int cols, rows, sheets;      // entries: columns from col0 on (around the end), rows from row0 on, sheets
};
__device__ __forceinline__ Span span_of(const int* n, int per_cta) {
  const long long plane = (long long)n[0] * n[1] * n[2];
  const long long first = blockIdx.x * (long long)per_cta;
  const int count = (int)min((long long)per_cta, plane - first);
  Span sp;
  const long long row = first / n[2];
  sp.col0 = (int)(first - row * n[2]);
  sp.sheet0 = (int)(row / n[1]);
  sp.row0 = (int)(row - (long long)sp.sheet0 * n[1]);
  sp.cols = min(per_cta, n[2]);
  sp.rows = (sp.col0 + count - 1) / n[2] + 1;
  sp.sheets = (sp.row0 + sp.rows - 1) / n[1] + 1;
  return sp;
}
// entry t of the table -> (dimension, index)
__device__ __forceinline__ void span_entry(const Span& sp, const int* n, int t, int& d, int& i) {
  if (t < sp.cols) { d = 2; i = sp.col0 + t; if (i >= n[2]) i -= n[2]; return; }
  t -= sp.cols;
  if (t < sp.rows) { d = 1; i = (sp.row0 + t) % n[1]; return; }
  d = 0; i = sp.sheet0 + t - sp.rows;
}
// position number `off` of the CTA -> its entries and its indices
__device__ __forceinline__ void span_locate(const Span& sp, const int* n, int off, int* entry, int* i) {
  const int c = sp.col0 + off, row = c / n[2];
  i[2] = c - row * n[2];
  entry[2] = off < sp.cols ? off : (i[2] >= sp.col0 ? i[2] - sp.col0 : i[2] - sp.col0 + n[2]);
  const int h = sp.row0 + row, sheet = h / n[1];
  i[1] = h - sheet * n[1];
  entry[1] = sp.cols + row;
  i[0] = sp.sheet0 + sheet;
  entry[0] = sp.cols + sp.rows + sheet;
}
constexpr int kMaxEntries(int per_cta) { return per_cta + 2 * (kThreads + 2); }

// planes that this CTA walks
__device__ __forceinline__ int planes_left(long long BC) { return (int)((BC - blockIdx.y + gridDim.y - 1) / gridDim.y); }

// V consecutive outputs of one row per thread (V divides the row, so that a pair of bf16 leaves as one word).
// I: offsets within a plane of x, 32 bits unless a plane is larger than that.
template <typename T, int ND, int V, typename I>
__global__ void __launch_bounds__(kThreads)
interp_fwd_kernel(const InterpGeom g, const T* __restrict__ x, T* __restrict__ y, long long BC) {
  using A = typename Acc<T>::type;
  __shared__ int s_i[2][kMaxEntries(kThreads * V)];
  __shared__ A s_w[2][kMaxEntries(kThreads * V)];
  const long long out_plane = (long long)g.out_local[0] * g.out_local[1] * g.out_local[2];
  const long long in_plane = (long long)g.in_local[0] * g.in_local[1] * g.in_local[2];
  const Span sp = span_of(g.out_local, (int)blockDim.x * V);
  for (int t = threadIdx.x; t < sp.cols + sp.rows + sp.sheets; t += blockDim.x) {
    int d, o, a[2];
    span_entry(sp, g.out_local, t, d, o);
    A lam;
    source_index<A>(g, d, o, a[0], a[1], lam);
    const A w[2] = {(A)1 - lam, lam};
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const bool in = a[s] >= 0 && a[s] < g.in_local[d];
      s_i[s][t] = in ? a[s] : 0;
      s_w[s][t] = in ? w[s] : (A)0;
    }
  }
  __syncthreads();
  const long long first = (blockIdx.x * (long long)blockDim.x + threadIdx.x) * V;
  if (first >= out_plane) return;
  int entry[3], o[3];
  span_locate(sp, g.out_local, (int)threadIdx.x * V, entry, o);
  constexpr int NR = 1 << (ND - 1);                // source rows (leading dimensions of extent 1 are not interpolated)
  I at[NR][V][2];
  Weight<A> wr[NR], wc[V][2];
  I col[V][2];
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int e = entry[2] + v < sp.cols ? entry[2] + v : entry[2] + v - sp.cols;   // (V > 1: the row goes on)
#pragma unroll
    for (int s = 0; s < 2; ++s) { col[v][s] = s_i[s][e]; wc[v][s].set(s_w[s][e]); }
  }
#pragma unroll
  for (int i = 0; i < NR; ++i) {
    const int s1 = i & 1, s0 = (i >> 1) & 1;
    const I row = ((I)s_i[s0][entry[0]] * g.in_local[1] + s_i[s1][entry[1]]) * g.in_local[2];
    wr[i].set((ND >= 3 ? s_w[s0][entry[0]] : (A)1) * (ND >= 2 ? s_w[s1][entry[1]] : (A)1));
#pragma unroll
    for (int v = 0; v < V; ++v) { at[i][v][0] = row + col[v][0]; at[i][v][1] = row + col[v][1]; }
  }
  // (pointers that step from plane to plane: a 64-bit product per plane and tensor costs more than the taps)
  const T* xb = x + blockIdx.y * in_plane;
  T* yo = y + blockIdx.y * out_plane + first;
  const long long xstep = gridDim.y * in_plane, ystep = gridDim.y * out_plane;
#pragma unroll (ND >= 3 ? 1 : 2)
  for (int left = planes_left(BC); left > 0; --left, xb += xstep, yo += ystep) {
    A acc[V];
#pragma unroll
    for (int v = 0; v < V; ++v) acc[v] = (A)0;
#pragma unroll
    for (int i = 0; i < NR; ++i) {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const A t = wc[v][1].add(wc[v][0].add((A)0, ld(xb + at[i][v][0])), ld(xb + at[i][v][1]));
        acc[v] = wr[i].add(acc[v], t);
      }
    }
    if constexpr (V == 2) *reinterpret_cast<uint32_t*>(yo) = dd::pack_bf16x2(acc[0], acc[1]);
    else st(yo, acc[0]);
  }
}

// weight with which output o (local) of dimension d takes input i (local)
template <typename A>
__device__ inline A adjoint_weight(const InterpGeom& g, int d, int o, int i) {
  int i0, i1;
  A lam;
  source_index<A>(g, d, o, i0, i1, lam);
  return (i0 == i ? (A)1 - lam : (A)0) + (i1 == i && lam != (A)0 ? lam : (A)0);
}

// Outputs that may take input i of dimension d: the inverse of the source coordinate at i - 1 and i + 1
// with one output of slack on either side (rounding), the tail for the last input (coordinates beyond it are
// clamped to it), clipped to the local outputs.
__host__ __device__ inline void adjoint_candidates(const InterpGeom& g, int d, int i, int& lo, int& hi) {
  const int ig = i + g.x_off[d], n_in = g.in_global[d], n_out = g.out_global[d];
  double step = g.scale[d], shift = 0.0;
  if (g.linear && g.align_corners) step = n_out > 1 ? (double)(n_in - 1) / (double)(n_out - 1) : 0.0;
  else if (g.linear) shift = 0.5;
  double first = 0.0, last = (double)(n_out - 1);
  if (step > 0.0) {
    if (ig > 0) first = floor(((double)(ig - 1) + shift) / step - shift) - 1.0;
    if (ig < n_in - 1) last = ceil(((double)(ig + 1) + shift) / step - shift) + 1.0;
  }
  const double b = (double)g.y_off[d], e = (double)g.y_off[d] + (double)g.out_local[d] - 1.0;
  first = fmin(fmax(first, b), e + 1.0);
  last = fmax(fmin(last, e), b - 1.0);
  lo = (int)first - g.y_off[d];
  hi = (int)last - g.y_off[d];
}

// Any number of outputs per dimension, weights worked out on the way: for positions with more than K of them.
template <typename T>
__device__ __noinline__ typename Acc<T>::type adjoint_any(const InterpGeom& g, const T* yb, const int* i, const int* lo,
                                                          const int* hi) {
  using A = typename Acc<T>::type;
  A acc = (A)0;
  for (int o0 = lo[0]; o0 <= hi[0]; ++o0) {
    const A w0 = adjoint_weight<A>(g, 0, o0, i[0]);
    if (w0 == (A)0) continue;
    for (int o1 = lo[1]; o1 <= hi[1]; ++o1) {
      const A w1 = adjoint_weight<A>(g, 1, o1, i[1]);
      if (w1 == (A)0) continue;
      A t = (A)0;
      for (int o2 = lo[2]; o2 <= hi[2]; ++o2)
        t += term<A>(adjoint_weight<A>(g, 2, o2, i[2]),
                     ld(yb + ((long long)o0 * g.out_local[1] + o1) * g.out_local[2] + o2));
      acc += term<A>(w0 * w1, t);
    }
  }
  return acc;
}

// Outputs of dimension d that take input i: lo .. lo + n - 1 with their weights; n = -1 where more than K do.
// WINDOW: the taps are moved to a window of K outputs that all exist (out_local[d] >= K), unused ones weigh zero.
template <typename A, int K, bool WINDOW>
__device__ __forceinline__ int adjoint_taps(const InterpGeom& g, int d, int i, int& lo, A* w) {
  int hi;
  adjoint_candidates(g, d, i, lo, hi);
  while (lo <= hi && adjoint_weight<A>(g, d, lo, i) == (A)0) ++lo;
  while (hi >= lo && adjoint_weight<A>(g, d, hi, i) == (A)0) --hi;
  const int n = hi - lo + 1;
  if (n <= 0) lo = 0;                            // nothing takes this input
  const int shift = WINDOW && lo + K > g.out_local[d] ? lo + K - g.out_local[d] : 0;
  lo -= shift;
  for (int j = 0; j < K; ++j) w[j] = j >= shift && j - shift < n ? adjoint_weight<A>(g, d, lo + j, i) : (A)0;
  return n > K ? -1 : n > 0 ? n : 0;
}

// K: outputs per dimension whose weights a thread keeps: up to five in registers, unrolled, from a table that the
// CTA fills together, as a window of outputs whose rows and columns lie at the same offsets for every thread; 32
// in a thread's own (local) memory, for scales above two and outputs smaller than the window.
template <typename T, int ND, int K>
__global__ void __launch_bounds__(kThreads)
interp_adjoint_kernel(const InterpGeom g, T* __restrict__ x, const T* __restrict__ y, long long BC) {
  using A = typename Acc<T>::type;
  constexpr bool TABLE = K <= 5;
  constexpr int E = TABLE ? kMaxEntries(kThreads) : 1;
  __shared__ int s_lo[E], s_n[E];
  __shared__ A s_w[TABLE ? K : 1][E];
  const long long out_plane = (long long)g.out_local[0] * g.out_local[1] * g.out_local[2];
  const long long in_plane = (long long)g.in_local[0] * g.in_local[1] * g.in_local[2];
  const Span sp = span_of(g.in_local, (int)blockDim.x);
  if constexpr (TABLE) {
    for (int t = threadIdx.x; t < sp.cols + sp.rows + sp.sheets; t += blockDim.x) {
      int d, i;
      span_entry(sp, g.in_local, t, d, i);
      A w[K];
      int lo = 0, n = 1;
      if (d < 3 - ND) {                           // a leading dimension of extent 1
#pragma unroll
        for (int j = 0; j < K; ++j) w[j] = (A)(j == 0 ? 1 : 0);
      } else {
        n = adjoint_taps<A, K, true>(g, d, i, lo, w);
      }
      s_lo[t] = lo;
      s_n[t] = n;
#pragma unroll
      for (int j = 0; j < K; ++j) s_w[j][t] = w[j];
    }
    __syncthreads();
  }
  const long long pos = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (pos >= in_plane) return;
  int entry[3], i[3], lo[3], n[3];
  A w[3][K];
  span_locate(sp, g.in_local, (int)threadIdx.x, entry, i);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if constexpr (TABLE) {
      lo[d] = s_lo[entry[d]];
      n[d] = s_n[entry[d]];
#pragma unroll
      for (int j = 0; j < K; ++j) w[d][j] = s_w[j][entry[d]];
    } else if (d < 3 - ND) {
      lo[d] = 0; n[d] = 1; w[d][0] = (A)1;
    } else {
      n[d] = adjoint_taps<A, K, false>(g, d, i[d], lo[d], w[d]);
    }
  }
  if (n[0] < 0 || n[1] < 0 || n[2] < 0) {
    int from[3], to[3];
    for (int d = 0; d < 3; ++d) adjoint_candidates(g, d, i[d], from[d], to[d]);
    for (long long bc = blockIdx.y; bc < BC; bc += gridDim.y)
      st(x + bc * in_plane + pos, adjoint_any<T>(g, y + bc * out_plane, i, from, to));
    return;
  }
  const long long base = ((long long)lo[0] * g.out_local[1] + lo[1]) * g.out_local[2] + lo[2];
  const long long s0 = (long long)g.out_local[1] * g.out_local[2];
  if constexpr (TABLE) {
    Weight<A> wc[K];
#pragma unroll
    for (int c = 0; c < K; ++c) wc[c].set(w[2][c]);
    const T* yb = y + blockIdx.y * out_plane + base;
    T* xo = x + blockIdx.y * in_plane + pos;
    const long long xstep = gridDim.y * in_plane, ystep = gridDim.y * out_plane;
#pragma unroll (ND >= 3 ? 1 : 2)
    for (int left = planes_left(BC); left > 0; --left, xo += xstep, yb += ystep) {
      A acc = (A)0;
#pragma unroll
      for (int a = 0; a < (ND >= 3 ? K : 1); ++a) {
        A sheet = (A)0;
#pragma unroll
        for (int b = 0; b < (ND >= 2 ? K : 1); ++b) {
          const T* row = yb + (a * s0 + (long long)b * g.out_local[2]);
          A t = (A)0;
#pragma unroll
          for (int c = 0; c < K; ++c) t = wc[c].add(t, ld(row + c));
          if (ND >= 2) { Weight<A> wb; wb.set(w[1][b]); sheet = wb.add(sheet, t); } else sheet = t;
        }
        if (ND >= 3) { Weight<A> wa; wa.set(w[0][a]); acc = wa.add(acc, sheet); } else acc = sheet;
      }
      st(xo, acc);
    }
  } else {
    for (long long bc = blockIdx.y; bc < BC; bc += gridDim.y) {
      const T* yb = y + bc * out_plane + base;
      A acc = (A)0;
      for (int a = 0; a < n[0]; ++a)
        for (int b = 0; b < n[1]; ++b) {
          A t = (A)0;
          for (int c = 0; c < n[2]; ++c) t += term<A>(w[2][c], ld(yb + a * s0 + (long long)b * g.out_local[2] + c));
          acc += term<A>(w[0][a] * w[1][b], t);
        }
      st(x + bc * in_plane + pos, acc);
    }
  }
}

// Two and three dimensions march along the leading one (rows, or sheets): what a sheet of the smaller tensor gives is
// the same for all the positions of the larger one before and behind it, so that a thread that holds one position of the
// other dimensions reads every sheet once instead of once per output.  What bounded the kernels above there was the
// number of loads: 8 per output of a volume and 64 per input in the adjoint (up-sampling by 1.5), now 3 and 27.
// In us, forward: [1, 32, 46^3] -> 69^3 in fp32 51 -> 42, [4, 72, 34^3] -> 68^3 in bf16 277 -> 186, [8, 64, 128, 128] -> 256^2 in
// bf16 76 -> 57.  The adjoint marches over volumes of 4-byte elements: the first of these 83 -> 58; in bf16 and over rows
// the loads of a sheet wait for each other more than they save (65 -> 109 for the last), but not where a window of five
// outputs is 125 of them: the second 407 -> 300 (909 with weights worked out on the way, as all of more than four were).
// Which tensors are walked so: march_forward, march_adjoint.
constexpr int kLead = 32;            // leading positions per segment, at most
constexpr int kLeadOut = 5 * kLead + 16;      // outputs that may take the inputs of a segment (adjoint)

struct Segments {
  int count, len;                    // over the leading positions, blockIdx.z
};

// dimensions behind the leading one, as the spans above take them
template <int ND> __device__ __forceinline__ void tail_of(const int* n, int* t) {
  t[0] = 1;
  t[1] = ND == 3 ? n[1] : 1;
  t[2] = n[2];
}

// V consecutive outputs of one row per thread (V divides the row, so that a pair of bf16 leaves as one word).
// I: offsets within a plane of x, 32 bits unless a plane is larger than that.
template <typename T, int ND, int V, typename I>
__global__ void __launch_bounds__(kThreads)
interp_fwd_march_kernel(const InterpGeom g, const T* __restrict__ x, T* __restrict__ y, long long BC, const Segments sg) {
  using A = typename Acc<T>::type;
  constexpr int LEAD = 3 - ND, NR = ND == 3 ? 2 : 1;
  __shared__ int s_i[2][kMaxEntries(kThreads * V)];
  __shared__ A s_w[2][kMaxEntries(kThreads * V)];
  __shared__ int l_i[2][kLead];
  __shared__ A l_w[2][kLead];
  int n[3];
  tail_of<ND>(g.out_local, n);
  const long long out_tail = (long long)n[1] * n[2];
  const long long in_tail = (long long)(ND == 3 ? g.in_local[1] : 1) * g.in_local[2];
  const Span sp = span_of(n, (int)blockDim.x * V);
  for (int t = threadIdx.x; t < sp.cols + sp.rows; t += blockDim.x) {
    int d, o, a[2];
    span_entry(sp, n, t, d, o);
    A lam = (A)0;
    if (ND == 2 && d == 1) { a[0] = a[1] = 0; }                 // (no such dimension behind the leading one)
    else source_index<A>(g, d, o, a[0], a[1], lam);
    const A w[2] = {(A)1 - lam, lam};
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const bool in = a[s] >= 0 && a[s] < g.in_local[d];
      s_i[s][t] = in ? a[s] : 0;
      s_w[s][t] = in ? w[s] : (A)0;
    }
  }
  __syncthreads();
  const long long first = (blockIdx.x * (long long)blockDim.x + threadIdx.x) * V;
  const bool mine = first < out_tail;
  int entry[3], o[3];
  span_locate(sp, n, mine ? (int)threadIdx.x * V : 0, entry, o);
  I at[NR][V][2];
  Weight<A> wr[NR], wc[V][2];
  I col[V][2];
#pragma unroll
  for (int v = 0; v < V; ++v) {
    const int e = entry[2] + v < sp.cols ? entry[2] + v : entry[2] + v - sp.cols;   // (V > 1: the row goes on)
#pragma unroll
    for (int s = 0; s < 2; ++s) { col[v][s] = s_i[s][e]; wc[v][s].set(s_w[s][e]); }
  }
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const I row = ND == 3 ? (I)s_i[r][entry[1]] * g.in_local[2] : (I)0;
    wr[r].set(ND == 3 ? s_w[r][entry[1]] : (A)1);
#pragma unroll
    for (int v = 0; v < V; ++v) { at[r][v][0] = row + col[v][0]; at[r][v][1] = row + col[v][1]; }
  }
  const long long xstep = gridDim.y * (in_tail * g.in_local[LEAD]), ystep = gridDim.y * (out_tail * g.out_local[LEAD]);
  for (int z = blockIdx.z; z < sg.count; z += gridDim.z) {
    const int o_first = z * sg.len, o_count = min(sg.len, g.out_local[LEAD] - o_first);
    __syncthreads();
    for (int t = threadIdx.x; t < o_count; t += blockDim.x) {
      int a[2];
      A lam;
      source_index<A>(g, LEAD, o_first + t, a[0], a[1], lam);
      const A w[2] = {(A)1 - lam, lam};
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const bool in = a[s] >= 0 && a[s] < g.in_local[LEAD];
        l_i[s][t] = in ? a[s] : 0;
        l_w[s][t] = in ? w[s] : (A)0;
      }
    }
    __syncthreads();
    if (!mine) continue;
    const T* xb = x + blockIdx.y * (in_tail * g.in_local[LEAD]);
    T* yb = y + blockIdx.y * (out_tail * g.out_local[LEAD]) + o_first * out_tail + first;
    for (int left = planes_left(BC); left > 0; --left, xb += xstep, yb += ystep) {
      A held[2][V];                                  // of the sheets number `sheet`
      int sheet[2] = {-1, -1};
      auto fetch = [&](int i, A (&v)[V]) {
        const T* xs = xb + i * in_tail;
#pragma unroll
        for (int j = 0; j < V; ++j) {
          v[j] = (A)0;
#pragma unroll
          for (int r = 0; r < NR; ++r) {
            const A t = wc[j][1].add(wc[j][0].add((A)0, ld(xs + at[r][j][0])), ld(xs + at[r][j][1]));
            v[j] = ND == 3 ? wr[r].add(v[j], t) : t;
          }
        }
      };
      T* yo = yb;
      for (int t = 0; t < o_count; ++t, yo += out_tail) {
        const int i0 = l_i[0][t], i1 = l_i[1][t];
        if (i0 != sheet[0]) {
          if (i0 == sheet[1]) {
#pragma unroll
            for (int j = 0; j < V; ++j) held[0][j] = held[1][j];
          } else {
            fetch(i0, held[0]);
          }
          sheet[0] = i0;
        }
        if (i1 != sheet[1]) {
          if (i1 == i0) {
#pragma unroll
            for (int j = 0; j < V; ++j) held[1][j] = held[0][j];
          } else {
            fetch(i1, held[1]);
          }
          sheet[1] = i1;
        }
        Weight<A> w0, w1;
        w0.set(l_w[0][t]);
        w1.set(l_w[1][t]);
        A acc[V];
#pragma unroll
        for (int j = 0; j < V; ++j) acc[j] = w1.add(w0.add((A)0, held[0][j]), held[1][j]);
        if constexpr (V == 2) *reinterpret_cast<uint32_t*>(yo) = dd::pack_bf16x2(acc[0], acc[1]);
        else st(yo, acc[0]);
      }
    }
  }
}

// K: outputs per dimension behind the leading one that take an input, at most (as above).
template <typename T, int K>
__global__ void __launch_bounds__(kThreads)
interp_adjoint_march_kernel(const InterpGeom g, T* __restrict__ x, const T* __restrict__ y, long long BC,
                            const Segments sg) {
  using A = typename Acc<T>::type;
  constexpr int E = kMaxEntries(kThreads);
  __shared__ int s_lo[E], s_n[E];
  __shared__ A s_w[K][E];
  __shared__ int l_a[kLeadOut];
  __shared__ A l_w[2][kLeadOut];
  int n[3];
  tail_of<3>(g.in_local, n);
  const long long in_tail = (long long)n[1] * n[2];
  const long long out_tail = (long long)g.out_local[1] * g.out_local[2];
  const int i_first = (int)blockIdx.z * sg.len, i_end = min(i_first + sg.len, g.in_local[0]);
  int o_first, o_last, skip;
  adjoint_candidates(g, 0, i_first, o_first, skip);
  adjoint_candidates(g, 0, i_end - 1, skip, o_last);
  const int o_count = min(o_last - o_first + 1, kLeadOut);      // (never cut: march_fits)
  const Span sp = span_of(n, (int)blockDim.x);
  for (int t = threadIdx.x; t < sp.cols + sp.rows; t += blockDim.x) {
    int d, i;
    span_entry(sp, n, t, d, i);
    A w[K];
    int lo = 0;
    const int taps = adjoint_taps<A, K, true>(g, d, i, lo, w);
    s_lo[t] = lo;
    s_n[t] = taps;
#pragma unroll
    for (int j = 0; j < K; ++j) s_w[j][t] = w[j];
  }
  for (int t = threadIdx.x; t < o_count; t += blockDim.x) {
    int a0, a1;
    A lam;
    source_index<A>(g, 0, o_first + t, a0, a1, lam);
    l_a[t] = a0;
    l_w[0][t] = (A)1 - lam;
    l_w[1][t] = a1 == a0 ? (A)0 : lam;
  }
  __syncthreads();
  const long long pos = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (pos >= in_tail) return;
  int entry[3], i[3];
  span_locate(sp, n, (int)threadIdx.x, entry, i);
  const T* yb = y + blockIdx.y * (out_tail * g.out_local[0]);
  T* xb = x + blockIdx.y * (in_tail * g.in_local[0]) + pos;
  const long long xstep = gridDim.y * (in_tail * g.in_local[0]), ystep = gridDim.y * (out_tail * g.out_local[0]);
  if (s_n[entry[2]] < 0 || s_n[entry[1]] < 0) {       // more than K outputs take this position
    for (int left = planes_left(BC); left > 0; --left, xb += xstep, yb += ystep)
      for (int il = i_first; il < i_end; ++il) {
        int from[3], to[3];
        i[0] = il;
        for (int d = 0; d < 3; ++d) adjoint_candidates(g, d, i[d], from[d], to[d]);
        st(xb + il * in_tail, adjoint_any<T>(g, yb, i, from, to));
      }
    return;
  }
  Weight<A> wc[K], wb[K];
#pragma unroll
  for (int c = 0; c < K; ++c) wc[c].set(s_w[c][entry[2]]);
#pragma unroll
  for (int b = 0; b < K; ++b) wb[b].set(s_w[b][entry[1]]);
  yb += o_first * out_tail + (long long)s_lo[entry[1]] * g.out_local[2] + s_lo[entry[2]];
  for (int left = planes_left(BC); left > 0; --left, xb += xstep, yb += ystep) {
    A acc0 = (A)0, acc1 = (A)0;                      // of the inputs `cur` and cur + 1
    int cur = i_first - 1;
    A ahead[K][K];                                  // of the next sheet, on its way while this one is added up
    auto fetch = [&](int t) {
#pragma unroll
      for (int b = 0; b < K; ++b)
#pragma unroll
        for (int c = 0; c < K; ++c) ahead[b][c] = ld(yb + t * out_tail + (long long)b * g.out_local[2] + c);
    };
    int t = 0;
    while (t < o_count && l_a[t] < i_first - 1) ++t;
    if (t < o_count) fetch(t);
    for (; t < o_count; ++t) {
      const int a = l_a[t];
      while (cur < a && cur < i_end) {
        if (cur >= i_first) st(xb + cur * in_tail, acc0);
        acc0 = acc1;
        acc1 = (A)0;
        ++cur;
      }
      if (cur >= i_end) break;
      A sum = (A)0;
      A v[K][K];
#pragma unroll
      for (int b = 0; b < K; ++b)
#pragma unroll
        for (int c = 0; c < K; ++c) v[b][c] = ahead[b][c];
      if (t + 1 < o_count) fetch(t + 1);
#pragma unroll
      for (int b = 0; b < K; ++b) {
        A q = (A)0;
#pragma unroll
        for (int c = 0; c < K; ++c) q = wc[c].add(q, v[b][c]);
        sum = wb[b].add(sum, q);
      }
      Weight<A> w0, w1;
      w0.set(l_w[0][t]);
      w1.set(l_w[1][t]);
      acc0 = w0.add(acc0, sum);
      acc1 = w1.add(acc1, sum);
    }
    for (; cur < i_end; ++cur) {
      if (cur >= i_first) st(xb + cur * in_tail, acc0);
      acc0 = acc1;
      acc1 = (A)0;
    }
  }
}

// Segments of the leading dimension and groups of planes.  A CTA's tables take as long as tens of sheets, so that a segment
// is long (kLead) unless that leaves SMs idle, and a CTA walks as many planes as about 2048 threads per SM allow.
inline dim3 march_grid(long long positions, int lead, long long BC, int threads, Segments& sg) {
  const long long bx = (positions + threads - 1) / threads;
  const long long want = 148LL * 2048 / threads;
  long long segs = std::max((lead + kLead - 1LL) / kLead, std::min((want + bx * BC - 1) / (bx * BC), (long long)(lead / 8)));
  sg.len = (int)((lead + segs - 1) / segs);
  sg.count = (lead + sg.len - 1) / sg.len;
  const long long each = std::max(BC * bx * sg.count / want, 1LL);       // planes of a CTA
  const long long by = std::min((BC + each - 1) / each, 65535LL);
  return dim3((unsigned)bx, (unsigned)by, (unsigned)std::min(sg.count, 65535));
}

// CTAs over positions x groups of planes: about sixteen CTAs per SM in all, so that a thread keeps its indices
// for as many planes as leave the GPU full
inline dim3 plane_grid(long long positions, long long BC, int threads) {
  const long long bx = (positions + threads - 1) / threads;
  long long by = (148LL * 16 + bx - 1) / bx;
  if (by > BC) by = BC;
  if (by > 65535) by = 65535;
  return dim3((unsigned)bx, (unsigned)by);
}
inline int plane_threads(long long positions) {
  return positions >= kThreads ? kThreads : (int)((positions + 31) / 32 * 32);
}

// Whether the outputs that may take the inputs of a segment fit the adjoint's table: between the ends of the dimension
// (len + 1) / step and a few, at the last input as many as lie beyond it.
inline bool march_fits(const InterpGeom& g, const Segments& sg, double step) {
  if (sg.count > 65535 || !(step > 0.0) || (sg.len + 1) / step + 8.0 > kLeadOut) return false;
  int lo, hi, skip;
  adjoint_candidates(g, 0, (sg.count - 1) * sg.len, lo, skip);
  adjoint_candidates(g, 0, g.in_local[0] - 1, skip, hi);
  return hi - lo < kLeadOut;
}

// Source step per output along dimension d (0: all outputs take the same).
inline double step_of(const InterpGeom& g, int d) {
  if (!(g.linear && g.align_corners)) return g.scale[d];
  return g.out_global[d] > 1 ? (double)(g.in_global[d] - 1) / (double)(g.out_global[d] - 1) : 0.0;
}

// Whether the forward walks sheets (or rows), of V outputs of esize bytes per thread.  That gains where a sheet is read by
// several outputs of the leading dimension, so not where that grows by less than 1.4 (size kept, rows of 256, 2^24 outputs in
// fp32: 1.15 times the time of the kernel above; halved, rows of 128 in bf16, 2^23: 1.6).  The threads of a CTA lie over one sheet: short
// rows leave lanes without one, and whole tensors beyond L2 hide loads by themselves, so that the kernel above is the faster one
// for rows.  Times the kernel's above, growing by 2 (by 1.5), outputs in all 2^20, 2^21, 2^23, 2^25:
//   rows in bf16    of 32 0.98 1.24 2.01 2.07 (0.99 1.35 2.22 2.66), 64 0.80 0.90 1.31 1.42 (0.77 0.96 1.46 1.77), 128 0.54 0.76 0.92 1.02
//                   (0.62 0.77 0.98 1.08), 160 0.58 0.61 0.84 0.80 (0.60 0.67 0.87 0.89), 256 0.49 0.51 0.72 0.72
//   rows in fp32    of 32 0.81 1.11 1.54 1.70, 64 0.62 0.86 1.06 1.39 (0.64 0.87 1.16 1.49), 128 0.66 0.77 0.96 1.03 (0.63 0.78 1.05
//                   1.15; 0.90 of 2^22), 384 0.60 0.67 0.93 1.21 (0.61 0.68 1.05 1.39), 512 0.52 0.58 0.80 1.00 (0.52 0.58 0.90 1.10);
//                   of 260, half the lanes of two CTAs, 2^22 (1.09)
//   sheets in bf16  of 6 x 6 1.24 - 1.26 1.06, 8 x 8 0.66 0.79 1.20 0.91 (0.68 0.84 1.31 1.10), 12 x 12 0.53 0.59 0.81 0.75 (0.60 0.66
//                   0.92 0.96), 32 x 32 0.51 0.59 0.72 0.62
//   sheets in fp32  of 6 x 6 0.98 - 1.07 1.18, 8 x 8 0.57 0.72 0.75 0.78 (0.63 0.74 0.81 0.91), 24 x 24 0.64 0.84 0.78 0.80 (0.65 0.88
//                   0.88 1.01); in fp64 - 0.90 0.93 1.01 (- 0.99 1.06 1.05)
// Below 2^20 the tables take longer than the loads (10^3: 3.5 and 6.7 us).
inline bool march_forward(const InterpGeom& g, int nd, long long tail, long long outputs, int V, int esize) {
  if (nd < 2 || outputs < (1 << 20) || step_of(g, 3 - nd) > 0.72) return false;
  const long long threads = tail / V, per_cta = plane_threads(threads), lanes = (threads + per_cta - 1) / per_cta * per_cta;
  const bool busy = threads * 5 >= lanes * 4;
  if (nd == 3) return threads >= 64 && (esize <= 4 || (busy && outputs < (1 << 22)));
  if (V == 2) return busy && (threads >= 72 || (threads >= 32 && outputs <= (1 << 21)));
  return busy && ((threads >= 128 && outputs < (3 << 21)) || (threads >= 64 && outputs <= (1 << 21)));
}

// Outputs of a row per thread: a pair of bf16, where a row is whole pairs, leaves as one word.
template <typename T>
inline int forward_vector(const InterpGeom& g, bool small, const T* y) {
  return std::is_same<T, __nv_bfloat16>::value && small && g.out_local[2] % 2 == 0 && (reinterpret_cast<uintptr_t>(y) & 3) == 0
             ? 2 : 1;
}

// Outputs per input and dimension that a thread of the adjoint keeps weights for (32: in its own memory), as a hint: a position
// that has more takes the slow way by itself.  per: of the dimension that has the most, where the ratio is no whole number.
// Five cost a table of their own: 0.3 to 0.5 of the time in three dimensions, 0.4 to 0.8 in two, in one 0.6 to 0.95 for rows of 100
// and more, but 1.1 to 1.4 for 12 to 40 inputs unless there are 2^22 outputs (0.8 to 0.98), in fp64 even then, and 1.2 for 3 x 14 and 4 x 4 x 4.
inline int adjoint_window(const InterpGeom& g, int nd, long long outputs, int esize, double* per) {
  double most = 1.0;
  int least = g.out_local[2];                       // the smallest extent must hold a whole window
  *per = 1.0;
  for (int d = 2; d >= 3 - nd; --d) {
    if (g.out_local[d] < least) least = g.out_local[d];
    const double step = step_of(g, d), n = step > 0.0 ? (g.linear ? 2.0 : 1.0) / step : (double)g.out_local[d];
    *per = std::max(*per, n);
    most = std::max(most, step > 0.0 ? std::ceil(n - 1e-9) : n);
  }
  const bool five = (long long)g.in_local[0] * g.in_local[1] * g.in_local[2] >= 80 ||
                    (esize <= 4 && (nd >= 2 || outputs >= (1 << 22)));
  return most <= 2.0 && least >= 2 ? 2 : most <= 3.0 && least >= 3 ? 3 : most <= 4.0 && least >= 4 ? 4
         : most <= 5.0 && least >= 5 && five ? 5 : 32;
}

// Whether the adjoint walks sheets, with K outputs per dimension that take an input, `per` of them where the ratio is no whole
// number.  Nearest takes one and gains nothing (grown by 2, 2^20 outputs 1.3 to 1.9 times the time of the kernel above).  Times
// the kernel's, in fp32, outputs in all 2^20, 2^21, 2^22, 2^23, 2^25:
//   halved (K = 2)          32 x 32 inputs 0.90 0.80 0.77 0.75 0.82, 20 x 20 1.02 0.99 1.08 1.09 0.94; size kept, 24 x 24 0.79 - 1.25 - 1.55
//   grown by 1.5 (K = 3)    7 x 7 0.60 0.82 1.02 1.27 1.20, 9 x 9 0.73 0.55 0.75 0.79 0.68, 16 x 16 0.78 0.56 0.81 0.98 1.17, 32 x 32 0.78 0.55
//                           0.77 0.92 1.09 (fp64 - 0.56 - 0.83 0.75)
//   grown by 2 (K = 4)      6 x 6 0.92 0.78 0.86 1.19 1.34, 7 x 7 0.88 0.68 0.81 0.91 0.98, 16 x 16 1.47 0.94 0.61 0.62 0.92
//   the same with corners   (K = 5), bf16 as well: 5 x 5 1.09 1.15 1.60 1.85 1.67, 16 x 16 1.41 0.88 0.60 0.74 0.81
inline bool march_adjoint(const InterpGeom& g, int K, double per, long long tail, long long outputs, int esize) {
  if (!g.linear || outputs < (1 << 20) || K > 5 || (esize < 4 && K != 5)) return false;
  if (K == 2) return tail >= 1024 && step_of(g, 0) >= 1.9;
  if (K == 3) return tail >= 81 && (esize == 8 || outputs <= (1 << 23));
  return tail >= 49 && (per < 3.4 || outputs >= (3 << 20));
}

template <typename T, int ND>
int run_cuda(int adjoint, const InterpGeom& g, T* x, T* y, long long BC, cudaStream_t s) {
  const long long in_plane = (long long)g.in_local[0] * g.in_local[1] * g.in_local[2];
  const long long out_plane = (long long)g.out_local[0] * g.out_local[1] * g.out_local[2];
  if (!adjoint) {
    if (BC * out_plane <= 0) return 0;
    // an empty slab of the input gives nothing to any output, and holds no element that the kernel could read with
    // weight zero
    if (in_plane <= 0) return (int)cudaMemsetAsync(y, 0, (size_t)(BC * out_plane) * sizeof(T), s);
    const bool small = in_plane < 0x7fffffffLL;
    const int V = forward_vector<T>(g, small, y);
    if constexpr (ND >= 2) {
      const long long tail = out_plane / g.out_local[3 - ND];
      if (march_forward(g, ND, tail, BC * out_plane, V, (int)sizeof(T))) {
        Segments sg;
        if constexpr (std::is_same<T, __nv_bfloat16>::value) {
          if (V == 2) {
            const int t = plane_threads(tail / 2);
            const dim3 grid = march_grid(tail / 2, g.out_local[3 - ND], BC, t, sg);
            interp_fwd_march_kernel<T, ND, 2, int><<<grid, t, 0, s>>>(g, x, y, BC, sg);
            return (int)cudaGetLastError();
          }
        }
        const int t = plane_threads(tail);
        const dim3 grid = march_grid(tail, g.out_local[3 - ND], BC, t, sg);
        if (small) interp_fwd_march_kernel<T, ND, 1, int><<<grid, t, 0, s>>>(g, x, y, BC, sg);
        else       interp_fwd_march_kernel<T, ND, 1, long long><<<grid, t, 0, s>>>(g, x, y, BC, sg);
        return (int)cudaGetLastError();
      }
    }
    if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      if (V == 2) {
        const int t = plane_threads(out_plane / 2);
        interp_fwd_kernel<T, ND, 2, int><<<plane_grid(out_plane / 2, BC, t), t, 0, s>>>(g, x, y, BC);
        return (int)cudaGetLastError();
      }
    }
    const int t = plane_threads(out_plane);
    if (small) interp_fwd_kernel<T, ND, 1, int><<<plane_grid(out_plane, BC, t), t, 0, s>>>(g, x, y, BC);
    else       interp_fwd_kernel<T, ND, 1, long long><<<plane_grid(out_plane, BC, t), t, 0, s>>>(g, x, y, BC);
    return (int)cudaGetLastError();
  }
  if (BC * in_plane <= 0) return 0;
  if (out_plane <= 0) return (int)cudaMemsetAsync(x, 0, (size_t)(BC * in_plane) * sizeof(T), s);
  double per;
  const int K = adjoint_window(g, ND, BC * out_plane, (int)sizeof(T), &per);
  if constexpr (ND == 3) {
    const long long tail = in_plane / g.in_local[0];
    const int t = plane_threads(tail);
    Segments sg;
    const dim3 grid = march_grid(tail, g.in_local[0], BC, t, sg);
    if (march_adjoint(g, K, per, tail, BC * out_plane, (int)sizeof(T)) && march_fits(g, sg, step_of(g, 0))) {
      if (K == 5) interp_adjoint_march_kernel<T, 5><<<grid, t, 0, s>>>(g, x, y, BC, sg);
      if constexpr (sizeof(T) >= 4) {
        if (K == 2)      interp_adjoint_march_kernel<T, 2><<<grid, t, 0, s>>>(g, x, y, BC, sg);
        else if (K == 3) interp_adjoint_march_kernel<T, 3><<<grid, t, 0, s>>>(g, x, y, BC, sg);
        else if (K == 4) interp_adjoint_march_kernel<T, 4><<<grid, t, 0, s>>>(g, x, y, BC, sg);
      }
      return (int)cudaGetLastError();
    }
  }
  const int t = plane_threads(in_plane);
  const dim3 grid = plane_grid(in_plane, BC, t);
  if (K == 2)      interp_adjoint_kernel<T, ND, 2><<<grid, t, 0, s>>>(g, x, y, BC);
  else if (K == 3) interp_adjoint_kernel<T, ND, 3><<<grid, t, 0, s>>>(g, x, y, BC);
  else if (K == 4) interp_adjoint_kernel<T, ND, 4><<<grid, t, 0, s>>>(g, x, y, BC);
  else if (K == 5) interp_adjoint_kernel<T, ND, 5><<<grid, t, 0, s>>>(g, x, y, BC);
  else             interp_adjoint_kernel<T, ND, 32><<<grid, t, 0, s>>>(g, x, y, BC);
  return (int)cudaGetLastError();
}

template <typename T, bool ADJOINT>
void interp_cpu(const InterpGeom& g, T* x, T* y, long long BC) {
  // parallel over batch*channel planes: the adjoint's scatter never crosses planes
#pragma omp parallel for schedule(static)
  for (long long bc = 0; bc < BC; ++bc)
    for (int o0 = 0; o0 < g.out_local[0]; ++o0)
      for (int o1 = 0; o1 < g.out_local[1]; ++o1)
        for (int o2 = 0; o2 < g.out_local[2]; ++o2) process_output<T, ADJOINT>(g, x, y, bc, o0, o1, o2);
}

template <typename T>
int run(int cuda, int adjoint, const InterpGeom& g, int nd, void* x, void* y, long long BC, void* stream) {
  T* xp = reinterpret_cast<T*>(x);
  T* yp = reinterpret_cast<T*>(y);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (cuda)
    return nd == 1 ? run_cuda<T, 1>(adjoint, g, xp, yp, BC, s)
                   : nd == 2 ? run_cuda<T, 2>(adjoint, g, xp, yp, BC, s) : run_cuda<T, 3>(adjoint, g, xp, yp, BC, s);
  if constexpr (std::is_same<T, __nv_bfloat16>::value) return DD_ERR_BAD_ARG;
  else {
    if (adjoint) interp_cpu<T, true>(g, xp, yp, BC); else interp_cpu<T, false>(g, xp, yp, BC);
    return 0;
  }
}

InterpGeom make_geom(int linear, int nd, const int* in_local, const int* out_local, const int* x_off, const int* y_off,
                     const int* in_global, const int* out_global, const double* scale, int align_corners) {
  InterpGeom g;
  for (int d = 0; d < 3; ++d) {
    const int s = d - (3 - nd);     // leading dims are padded with extent 1
    if (s < 0) {
      g.in_local[d] = g.out_local[d] = g.in_global[d] = g.out_global[d] = 1;
      g.x_off[d] = g.y_off[d] = 0;
      g.scale[d] = 1.0;
    } else {
      g.in_local[d] = in_local[s]; g.out_local[d] = out_local[s];
      g.x_off[d] = x_off[s]; g.y_off[d] = y_off[s];
      g.in_global[d] = in_global[s]; g.out_global[d] = out_global[s];
      g.scale[d] = scale[s];
    }
  }
  g.align_corners = align_corners;
  g.linear = linear;
  return g;
}

}  // namespace

// nd in 1..3; all int arrays have nd entries; scale[d] = source step per output
// index (1 / scale_factor, or in_global / out_global).  Forward: y = I(x).
// Adjoint: x = I^T(y) (on the CPU x += I^T(y) into an x that the caller has zeroed).
// dtype: 0 fp32, 1 fp64, 2 bf16 (CUDA only; weights and sums in fp32).
DD_API int dd_interpolate(int cuda, int linear, int adjoint, int dtype, int nd, void* x, void* y, long long BC,
                          const int* in_local, const int* out_local, const int* x_off, const int* y_off,
                          const int* in_global, const int* out_global, const double* scale, int align_corners,
                          void* stream) {
  if (nd < 1 || nd > 3 || BC < 0) return DD_ERR_BAD_ARG;
  const InterpGeom g = make_geom(linear, nd, in_local, out_local, x_off, y_off, in_global, out_global, scale, align_corners);
  // (an empty tensor has no address, and so has one without storage, which must not reach a kernel)
  long long n_in = BC, n_out = BC;
  for (int d = 0; d < 3; ++d) { n_in *= g.in_local[d]; n_out *= g.out_local[d]; }
  if ((x == nullptr && n_in > 0) || (y == nullptr && n_out > 0)) return DD_ERR_BAD_ARG;
  if (dtype == 0) return run<float>(cuda, adjoint, g, nd, x, y, BC, stream);
  if (dtype == 1) return run<double>(cuda, adjoint, g, nd, x, y, BC, stream);
  return run<__nv_bfloat16>(cuda, adjoint, g, nd, x, y, BC, stream);
}

// Whether the call above walks sheets (or rows) on the GPU, for tests.
DD_API int dd_interpolate_marches(int linear, int adjoint, int dtype, int nd, long long BC, const int* in_local,
                                  const int* out_local, const int* x_off, const int* y_off, const int* in_global,
                                  const int* out_global, const double* scale, int align_corners) {
  if (nd < 1 || nd > 3) return 0;
  const InterpGeom g = make_geom(linear, nd, in_local, out_local, x_off, y_off, in_global, out_global, scale, align_corners);
  const long long in_plane = (long long)g.in_local[0] * g.in_local[1] * g.in_local[2];
  const long long out_plane = (long long)g.out_local[0] * g.out_local[1] * g.out_local[2];
  if (in_plane <= 0 || out_plane <= 0) return 0;
  const int esize = dtype == 0 ? 4 : dtype == 1 ? 8 : 2;
  if (!adjoint) {
    const bool pairs = dtype == 2 && in_plane < 0x7fffffffLL && g.out_local[2] % 2 == 0;
    return nd >= 2 && march_forward(g, nd, out_plane / g.out_local[3 - nd], BC * out_plane, pairs ? 2 : 1, esize);
  }
  double per;
  const int K = adjoint_window(g, nd, BC * out_plane, esize, &per);
  const long long tail = in_plane / g.in_local[0];
  Segments sg;
  march_grid(tail, g.in_local[0], BC, plane_threads(tail), sg);
  return nd == 3 && march_adjoint(g, K, per, tail, BC * out_plane, esize) && march_fits(g, sg, step_of(g, 0));
}
