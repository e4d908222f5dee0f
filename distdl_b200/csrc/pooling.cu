// Local arithmetic of the distributed pooling layers: average and max pooling of
// [planes, n0, n1, n2] tensors (planes = batch x channels; 1-D and 2-D pooling use leading
// extents of 1), fp32 or bf16, no padding (the layer pads at the global boundary and
// exchanges halos first, nn/pooling.py).  The input may be a strided view (the cropped
// interior of the halo-exchanged tensor), so the crop costs no copy; outputs are contiguous.
// The reference calls torch.nn.functional.{avg,max}_pool{1,2,3}d on a contiguous crop here
// (src/distdl/nn/pooling.py:150-170).
//
//   forward : one thread per output element walks its window (dilated for max pooling);
//             max pooling also records the input position of the maximum (the first of equal
//             values wins, a NaN wins over everything, as in PyTorch).
//   backward: one thread per INPUT element gathers from the outputs whose windows cover it
//             (no atomics, deterministic); dx is contiguous with the shape of the view.
#include "common.cuh"

using namespace dd;

namespace {

struct PoolGeom {
  long long planes;
  int in[3], out[3], k[3], s[3], d[3];
  long long xs_plane, xs[3];      // element strides of the input view
};

template <typename T> __device__ __forceinline__ float pf(T v);
template <> __device__ __forceinline__ float pf<float>(float v) { return v; }
template <> __device__ __forceinline__ float pf<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
// planes that this CTA walks
__device__ __forceinline__ int planes_left(const PoolGeom& g) {
  return (int)((g.planes - blockIdx.y + gridDim.y - 1) / gridDim.y);
}
template <typename T> __device__ __forceinline__ T pt(float v);
template <> __device__ __forceinline__ float pt<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 pt<__nv_bfloat16>(float v) { return __float2bfloat16(v); }

// Both kernels are bound by memory once the index arithmetic is out of the way, so a thread fixes one
// position of the plane, decodes it once (64-bit divisions) and walks the planes with it; windows of the
// common sizes are unrolled so that their loads are in flight together (K / C = 0: sizes at run time).
// [8, 64, 256, 256] bf16, max 2x2 stride 2: forward 119 -> 26 us, backward 585 -> 28 us;
// [1, 32, 93, 93, 93] fp32, average 3^3 stride 2: 130 -> 44 and 725 -> 61 us (before: every
// element decoded by itself).
// UNIT: neighbours along the last dimension of the window are neighbours in memory, and a plane's offsets fit
// 32 bits, so that a row of the window is one address.
template <typename T, bool MAX, int K0, int K1, int K2, bool UNIT>
__global__ void __launch_bounds__(256)
pool_fwd_kernel(const T* __restrict__ x, T* __restrict__ y, int* __restrict__ arg, const PoolGeom g, float inv_vol) {
  const long long per_plane = (long long)g.out[0] * g.out[1] * g.out[2];
  const long long pos = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (pos >= per_plane) return;
  long long r = pos;
  const int o2 = (int)(r % g.out[2]); r /= g.out[2];
  const int o1 = (int)(r % g.out[1]), o0 = (int)(r / g.out[1]);
  const int k0 = K0 ? K0 : g.k[0], k1 = K1 ? K1 : g.k[1], k2 = K2 ? K2 : g.k[2];
  const int first = (o0 * g.s[0] * g.in[1] + o1 * g.s[1]) * g.in[2] + o2 * g.s[2];
  const long long off = (long long)o0 * g.s[0] * g.xs[0] + (long long)o1 * g.s[1] * g.xs[1] +
                        (long long)o2 * g.s[2] * g.xs[2];
  const long long st0 = g.d[0] * g.xs[0], st1 = g.d[1] * g.xs[1], st2 = g.d[2] * g.xs[2];
  const int ix0 = g.d[0] * g.in[1] * g.in[2], ix1 = g.d[1] * g.in[2], ix2 = g.d[2];
  const T* xp = x + blockIdx.y * g.xs_plane + off;
  T* yp = y + blockIdx.y * per_plane + pos;
  int* ap = MAX ? arg + blockIdx.y * per_plane + pos : nullptr;
  const long long xstep = gridDim.y * g.xs_plane, ystep = gridDim.y * per_plane;
#pragma unroll (K0 * K1 * K2 == 0 || K0 * K1 * K2 > 9 ? 1 : 4)
  for (int left = planes_left(g); left > 0; --left, xp += xstep, yp += ystep, ap += MAX ? ystep : 0) {
    float acc = MAX ? -INFINITY : 0.f;
    int best = first;
#pragma unroll
    for (int a = 0; a < k0; ++a)
#pragma unroll
      for (int b = 0; b < k1; ++b)
#pragma unroll
        for (int c = 0; c < k2; ++c) {
          const float v = pf<T>(UNIT ? xp[a * (int)st0 + b * (int)st1 + c] : xp[a * st0 + b * st1 + c * st2]);
          if (MAX) {
            if (v > acc || v != v) { acc = v; best = first + a * ix0 + b * ix1 + c * ix2; }
          } else {
            acc += v;
          }
        }
    *yp = pt<T>(MAX ? acc : acc * inv_vol);
    if (MAX) *ap = best;
  }
}

// outputs o with o * s + a * d == i for some 0 <= a < k, o in [0, n_out): the range of candidates
__device__ __forceinline__ void cover(int i, int k, int s, int d, int n_out, int& lo, int& hi) {
  const int first = i - (k - 1) * d;                         // smallest window start that still reaches i
  lo = first <= 0 ? 0 : (first + s - 1) / s;
  hi = i / s;
  if (hi > n_out - 1) hi = n_out - 1;
}

// C0, C1, C2: most windows that cover an input along each dimension (without dilation), 0 = at run time
template <typename T, bool MAX, int C0, int C1, int C2>
__global__ void __launch_bounds__(256)
pool_bwd_kernel(const T* __restrict__ dy, const int* __restrict__ arg, T* __restrict__ dx, const PoolGeom g,
                float inv_vol) {
  const long long per_plane = (long long)g.in[0] * g.in[1] * g.in[2];
  const long long out_plane = (long long)g.out[0] * g.out[1] * g.out[2];
  const long long pos = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (pos >= per_plane) return;
  const int here = (int)pos;
  const int i2 = here % g.in[2], i1 = here / g.in[2] % g.in[1], i0 = here / g.in[2] / g.in[1];
  int lo0, hi0, lo1, hi1, lo2, hi2;
  cover(i0, g.k[0], g.s[0], g.d[0], g.out[0], lo0, hi0);
  cover(i1, g.k[1], g.s[1], g.d[1], g.out[1], lo1, hi1);
  cover(i2, g.k[2], g.s[2], g.d[2], g.out[2], lo2, hi2);
  const long long base = ((long long)lo0 * g.out[1] + lo1) * g.out[2] + lo2;
  const long long row0 = (long long)g.out[1] * g.out[2];
  const int n0 = hi0 - lo0 + 1, n1 = hi1 - lo1 + 1, n2 = hi2 - lo2 + 1;
  const T* dyp = dy + blockIdx.y * out_plane + base;
  const int* ap = MAX ? arg + blockIdx.y * out_plane + base : nullptr;
  T* dxp = dx + blockIdx.y * per_plane + pos;
  const long long istep = gridDim.y * per_plane, ostep = gridDim.y * out_plane;
#pragma unroll (C0 * C1 * C2 == 0 || C0 * C1 * C2 > 4 ? 1 : 4)
  for (int left = planes_left(g); left > 0; --left, dyp += ostep, ap += MAX ? ostep : 0, dxp += istep) {
    float acc = 0.f;
    if constexpr (C0 > 0) {
#pragma unroll
      for (int a = 0; a < C0; ++a)
#pragma unroll
        for (int b = 0; b < C1; ++b)
#pragma unroll
          for (int c = 0; c < C2; ++c)
            if (a < n0 && b < n1 && c < n2) {
              const long long o = a * row0 + (long long)b * g.out[2] + c;
              const float v = pf<T>(dyp[o]);
              if (!MAX || ap[o] == here) acc += v;
            }
    } else {
      for (int a = 0; a < n0; ++a) {
        if ((i0 - (lo0 + a) * g.s[0]) % g.d[0]) continue;
        for (int b = 0; b < n1; ++b) {
          if ((i1 - (lo1 + b) * g.s[1]) % g.d[1]) continue;
          for (int c = 0; c < n2; ++c) {
            if ((i2 - (lo2 + c) * g.s[2]) % g.d[2]) continue;
            const long long o = a * row0 + (long long)b * g.out[2] + c;
            if (!MAX || ap[o] == here) acc += pf<T>(dyp[o]);
          }
        }
      }
    }
    *dxp = pt<T>(MAX ? acc : acc * inv_vol);
  }
}

// Windows of 2 at stride 2 along the last dimension that tile it: two neighbouring inputs belong to the same
// outputs, so a thread takes the pair: one position, one argument and one gradient for two results that leave
// together.  C0, C1 as above (1 or at run time).
template <typename T, bool MAX, int C0, int C1>
__global__ void __launch_bounds__(256)
pool_bwd_pair_kernel(const T* __restrict__ dy, const int* __restrict__ arg, T* __restrict__ dx, const PoolGeom g,
                     float inv_vol) {
  const long long per_plane = (long long)g.in[0] * g.in[1] * g.in[2];
  const long long out_plane = (long long)g.out[0] * g.out[1] * g.out[2];
  const long long pos = 2 * (blockIdx.x * (long long)blockDim.x + threadIdx.x);
  if (pos >= per_plane) return;
  const int here = (int)pos;
  const int i2 = here % g.in[2], i1 = here / g.in[2] % g.in[1], i0 = here / g.in[2] / g.in[1];
  int lo0, hi0, lo1, hi1;
  cover(i0, g.k[0], g.s[0], 1, g.out[0], lo0, hi0);
  cover(i1, g.k[1], g.s[1], 1, g.out[1], lo1, hi1);
  const long long base = ((long long)lo0 * g.out[1] + lo1) * g.out[2] + (i2 >> 1);
  const long long row0 = (long long)g.out[1] * g.out[2];
  const int n0 = hi0 - lo0 + 1, n1 = hi1 - lo1 + 1;
  const T* dyp = dy + blockIdx.y * out_plane + base;
  const int* ap = MAX ? arg + blockIdx.y * out_plane + base : nullptr;
  T* d = dx + blockIdx.y * per_plane + pos;
  const long long istep = gridDim.y * per_plane, ostep = gridDim.y * out_plane;
#pragma unroll (C0 == 1 && C1 == 1 ? 4 : 1)
  for (int left = planes_left(g); left > 0; --left, dyp += ostep, ap += MAX ? ostep : 0, d += istep) {
    float a0 = 0.f, a1 = 0.f;
    for (int a = 0; a < (C0 ? C0 : n0); ++a)
      for (int b = 0; b < (C1 ? C1 : n1); ++b)
        if (a < n0 && b < n1) {
          const long long o = a * row0 + (long long)b * g.out[2];
          const float v = pf<T>(dyp[o]);
          if (MAX) {
            const int best = ap[o];
            if (best == here) a0 += v;
            if (best == here + 1) a1 += v;
          } else {
            a0 += v;
            a1 += v;
          }
        }
    if (!MAX) { a0 *= inv_vol; a1 *= inv_vol; }
    if constexpr (sizeof(T) == 2) *reinterpret_cast<uint32_t*>(d) = pack_bf16x2(a0, a1);
    else *reinterpret_cast<float2*>(d) = make_float2(a0, a1);
  }
}

int fill(PoolGeom& g, long long planes, const int* in, const int* out, const int* k, const int* s, const int* d,
         long long xs_plane, const long long* xs) {
  if (planes <= 0) return DD_ERR_BAD_ARG;
  g.planes = planes;
  g.xs_plane = xs_plane;
  for (int i = 0; i < 3; ++i) {
    if (in[i] <= 0 || out[i] <= 0 || k[i] <= 0 || s[i] <= 0 || d[i] <= 0) return DD_ERR_BAD_ARG;
    if ((long long)(out[i] - 1) * s[i] + (long long)(k[i] - 1) * d[i] >= in[i]) return DD_ERR_BAD_ARG;   // window leaves the input
    g.in[i] = in[i]; g.out[i] = out[i]; g.k[i] = k[i]; g.s[i] = s[i]; g.d[i] = d[i];
    g.xs[i] = xs ? xs[i] : 0;
  }
  if ((long long)in[0] * in[1] * in[2] > 0x7fffffffLL) return DD_ERR_TOO_LARGE;   // window positions are int32
  return 0;
}

// CTAs over positions x groups of planes: about sixteen CTAs per SM in all, so that a thread keeps its
// position for as many planes as leave the GPU full; small planes get a small CTA
int threads_for(long long positions) { return positions >= 256 ? 256 : (int)((positions + 31) / 32 * 32); }
dim3 grid_for(long long positions, long long planes) {
  const int t = threads_for(positions);
  const long long bx = (positions + t - 1) / t;
  long long by = (148LL * 16 + bx - 1) / bx;
  if (by > planes) by = planes;
  if (by > 65535) by = 65535;
  return dim3((unsigned)bx, (unsigned)by);
}

template <typename T, bool MAX>
void launch_fwd(const void* x, void* y, int* arg, const PoolGeom& g, float inv, cudaStream_t st) {
  const long long n = (long long)g.out[0] * g.out[1] * g.out[2];
  const dim3 grid = grid_for(n, g.planes);
  const int t = threads_for(n), *k = g.k;
  const T* xp = reinterpret_cast<const T*>(x);
  T* yp = reinterpret_cast<T*>(y);
  long long reach = 0;
  for (int i = 0; i < 3; ++i) reach += (long long)(g.in[i] - 1) * (g.xs[i] < 0 ? -g.xs[i] : g.xs[i]);
  const bool unit = g.xs[2] * g.d[2] == 1 && reach < 0x7fffffffLL;
#define DD_POOL_FWD(A, B, C) do { \
    if (unit) pool_fwd_kernel<T, MAX, A, B, C, true><<<grid, t, 0, st>>>(xp, yp, arg, g, inv); \
    else      pool_fwd_kernel<T, MAX, A, B, C, false><<<grid, t, 0, st>>>(xp, yp, arg, g, inv); } while (0)
  if (k[0] == 1 && k[1] == 2 && k[2] == 2)      DD_POOL_FWD(1, 2, 2);
  else if (k[0] == 1 && k[1] == 3 && k[2] == 3) DD_POOL_FWD(1, 3, 3);
  else if (k[0] == 2 && k[1] == 2 && k[2] == 2) DD_POOL_FWD(2, 2, 2);
  else if (k[0] == 3 && k[1] == 3 && k[2] == 3) DD_POOL_FWD(3, 3, 3);
  else                                          DD_POOL_FWD(0, 0, 0);
}

#undef DD_POOL_FWD

template <typename T, bool MAX>
void launch_bwd(const void* dy, const int* arg, void* dx, const PoolGeom& g, float inv, cudaStream_t st) {
  const long long n = (long long)g.in[0] * g.in[1] * g.in[2];
  const dim3 grid = grid_for(n, g.planes);
  const int t = threads_for(n);
  const T* dyp = reinterpret_cast<const T*>(dy);
  T* dxp = reinterpret_cast<T*>(dx);
  int c[3];
  bool dilated = false;
  for (int i = 0; i < 3; ++i) { c[i] = (g.k[i] + g.s[i] - 1) / g.s[i]; dilated = dilated || (g.d[i] != 1 && g.k[i] > 1); }
  const int most = c[0] > c[1] ? (c[0] > c[2] ? c[0] : c[2]) : (c[1] > c[2] ? c[1] : c[2]);
  const bool pair = g.k[2] == 2 && g.s[2] == 2 && !dilated && g.in[2] == 2 * g.out[2] &&
                    (reinterpret_cast<uintptr_t>(dx) & 7) == 0;
  if (pair) {
    const dim3 half = grid_for(n / 2, g.planes);
    const int th = threads_for(n / 2);
    if (c[0] == 1 && c[1] == 1) pool_bwd_pair_kernel<T, MAX, 1, 1><<<half, th, 0, st>>>(dyp, arg, dxp, g, inv);
    else                        pool_bwd_pair_kernel<T, MAX, 0, 0><<<half, th, 0, st>>>(dyp, arg, dxp, g, inv);
    return;
  }
  if (dilated || most > 3) pool_bwd_kernel<T, MAX, 0, 0, 0><<<grid, t, 0, st>>>(dyp, arg, dxp, g, inv);
  else if (most == 1)      pool_bwd_kernel<T, MAX, 1, 1, 1><<<grid, t, 0, st>>>(dyp, arg, dxp, g, inv);
  else if (most == 2 && c[0] == 1) pool_bwd_kernel<T, MAX, 1, 2, 2><<<grid, t, 0, st>>>(dyp, arg, dxp, g, inv);
  else if (most == 2)      pool_bwd_kernel<T, MAX, 2, 2, 2><<<grid, t, 0, st>>>(dyp, arg, dxp, g, inv);
  else if (c[0] == 1)      pool_bwd_kernel<T, MAX, 1, 3, 3><<<grid, t, 0, st>>>(dyp, arg, dxp, g, inv);
  else                     pool_bwd_kernel<T, MAX, 3, 3, 3><<<grid, t, 0, st>>>(dyp, arg, dxp, g, inv);
}

}  // namespace

// dtype: 0 = bf16, 1 = fp32; is_max: 0 = average (divides by the window volume), 1 = max.
// x: strided view [planes, in0, in1, in2] (xs_plane / xs: element strides); y: contiguous
// [planes, out0, out1, out2]; arg (max only): int32, same shape as y.
DD_API int dd_pool_fwd(const void* x, void* y, int* arg, long long planes, const int* in, const int* out, const int* k,
                       const int* s, const int* d, long long xs_plane, const long long* xs, int is_max, int dtype,
                       void* stream) {
  PoolGeom g;
  int r = fill(g, planes, in, out, k, s, d, xs_plane, xs);
  if (r) return r;
  if (x == nullptr || y == nullptr || (is_max && arg == nullptr)) return DD_ERR_BAD_ARG;
  const float inv = 1.f / ((float)k[0] * k[1] * k[2]);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (dtype == 0) { if (is_max) launch_fwd<__nv_bfloat16, true>(x, y, arg, g, inv, st); else launch_fwd<__nv_bfloat16, false>(x, y, arg, g, inv, st); }
  else            { if (is_max) launch_fwd<float, true>(x, y, arg, g, inv, st); else launch_fwd<float, false>(x, y, arg, g, inv, st); }
  return (int)cudaGetLastError();
}

// dy / arg: contiguous [planes, out...]; dx: contiguous [planes, in...] (the shape of the view x was).
DD_API int dd_pool_bwd(const void* dy, const int* arg, void* dx, long long planes, const int* in, const int* out,
                       const int* k, const int* s, const int* d, int is_max, int dtype, void* stream) {
  PoolGeom g;
  int r = fill(g, planes, in, out, k, s, d, 0, nullptr);
  if (r) return r;
  if (dy == nullptr || dx == nullptr || (is_max && arg == nullptr)) return DD_ERR_BAD_ARG;
  const float inv = 1.f / ((float)k[0] * k[1] * k[2]);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (dtype == 0) { if (is_max) launch_bwd<__nv_bfloat16, true>(dy, arg, dx, g, inv, st); else launch_bwd<__nv_bfloat16, false>(dy, arg, dx, g, inv, st); }
  else            { if (is_max) launch_bwd<float, true>(dy, arg, dx, g, inv, st); else launch_bwd<float, false>(dy, arg, dx, g, inv, st); }
  return (int)cudaGetLastError();
}
