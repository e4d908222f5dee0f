// Local arithmetic of the distributed batch norm on [batch, feature, rest...] tensors
// (contiguous, fp32 or bf16): per-feature reductions and the per-feature affine map.
// The layer (nn/batchnorm.py) exchanges the per-feature sums between workers with the
// SumReduce / Broadcast primitives; these kernels stand where the reference calls
// tensor.sum / elementwise PyTorch ops around those primitives
// (src/distdl/nn/batchnorm.py:306-360).
//
//   bn_reduce:  out[f]   (+)= sum over (b, r) of  u           u = x                (mode 0)
//               out2[f]  (+)= sum over (b, r) of  u * u       u = x - shift[f]     (mode 1)
//                                                 dy, dy * (x - shift[f])          (mode 2: out, out2)
//   bn_affine:  y = a[f] * (x - m[f]) + c[f]  (+ e[f] * z)   with optional second input z
// and, where one worker holds the whole batch (nothing to exchange between the passes), the layer's passes fused:
//   bn_train_fwd: mean and variance in ONE read of x, running statistics, y        (3 launches)
//   bn_train_bwd: sum dy, sum dy (x - mean) in one read, then dx through the statistics, dgamma, dbeta  (3 launches)
//
// All of them are bound by memory: 16-byte loads and stores on the 16-byte grid of the WHOLE tensor (the
// layouts agree, so a unit of one is a unit of all); the units that a plane [b, f, :] shares with its
// neighbours are taken element by element, so that any extent of `rest` runs vectorised.  [8, 64, 256, 256]
// bf16, forward + backward: 920 -> 112 us; [1, 32, 93, 93, 93] fp32: 740 -> 160 us (before: scalar loads
// with a 64-bit division per element, three reductions and five element-wise passes).
#include "common.cuh"

using namespace dd;

namespace {

constexpr int kBnThreads = 256;

template <typename T> __device__ __forceinline__ float to_f(T v);
template <> __device__ __forceinline__ float to_f<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16(v); }
__device__ __forceinline__ float load_as(const void* p, int dtype, int i) {
  return dtype == 0 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i]) : reinterpret_cast<const float*>(p)[i];
}
__device__ __forceinline__ float round_as(float v, int dtype) {
  return dtype == 0 ? __bfloat162float(__float2bfloat16(v)) : v;
}
__device__ __forceinline__ void store_as(void* p, int dtype, int i, float v) {
  if (dtype == 0) reinterpret_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16(v);
  else reinterpret_cast<float*>(p)[i] = v;
}

// VEC consecutive elements (16 bytes when VEC > 1; `p` is then 16-byte aligned)
template <typename T, int VEC>
__device__ __forceinline__ void load_unit(const T* __restrict__ p, float* v) {
  if constexpr (VEC == 1) {
    v[0] = to_f<T>(p[0]);
  } else {
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(p));
    if constexpr (sizeof(T) == 4) {
      v[0] = __uint_as_float(u.x); v[1] = __uint_as_float(u.y); v[2] = __uint_as_float(u.z); v[3] = __uint_as_float(u.w);
    } else {
      const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
      v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
    }
  }
}
template <typename T, int VEC>
__device__ __forceinline__ void store_unit(T* p, const float* v) {
  if constexpr (VEC == 1) {
    p[0] = from_f<T>(v[0]);
  } else if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<uint4*>(p) = make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]),
                                              __float_as_uint(v[3]));
  } else {
    *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]),
                                              pack_bf16x2(v[6], v[7]));
  }
}

// How the CTAs of a reduction share one feature: tpb threads side by side on the units of a plane, 256 / tpb
// planes at a time; `su` CTAs along the plane, `sb` over the batch.
struct Split {
  int tpb, su, sb;
};

// Visits the elements of feature f that this thread owns: whole units through full(offset), the elements of
// units at a plane's ends through one(offset).
template <int VEC, typename Full, typename One>
__device__ __forceinline__ void visit(int f, int B, int F, long long R, const Split& sp, Full full, One one) {
  const int tx = threadIdx.x % sp.tpb, ty = threadIdx.x / sp.tpb;
  const int rows = kBnThreads / sp.tpb;
  const int cu = blockIdx.y % sp.su, cb = blockIdx.y / sp.su;
  for (int b = cb * rows + ty; b < B; b += sp.sb * rows) {
    const long long p0 = ((long long)b * F + f) * R, p1 = p0 + R;
    const long long last = (p1 - 1) / VEC;
#pragma unroll 2
    for (long long u = p0 / VEC + cu * sp.tpb + tx; u <= last; u += (long long)sp.su * sp.tpb) {
      const long long e = u * VEC;
      if (VEC == 1 || (e >= p0 && e + VEC <= p1)) {
        full(e);
      } else {
        for (int i = 0; i < VEC; ++i)
          if (e + i >= p0 && e + i < p1) one(e + i);
      }
    }
  }
}

__device__ __forceinline__ float block_sum_bn(float v, float* red) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (lane < (kBnThreads >> 5)) ? red[lane] : 0.f;
  return warp_sum(t);
}

// grid = (F, su * sb).  PARTIALS: every CTA writes its two sums to out[(f * gridDim.y + split) * 2] (for a
// kernel that adds them up in order); otherwise it adds them to out[f] / out2[f] with one atomicAdd each.
template <typename T, int VEC, bool PARTIALS>
__global__ void __launch_bounds__(kBnThreads)
bn_reduce_kernel(const T* __restrict__ x, const T* __restrict__ dy, const float* __restrict__ shift, int B, int F,
                 long long R, int mode, Split sp, float* __restrict__ out, float* __restrict__ out2) {
  __shared__ float red[32];
  const int f = blockIdx.x;
  const float sh = (mode != 0 && shift != nullptr) ? shift[f] : 0.f;
  float a1 = 0.f, a2 = 0.f;
  if (mode == 2) {
    visit<VEC>(f, B, F, R, sp,
               [&](long long e) {
                 float u[VEC], g[VEC];
                 load_unit<T, VEC>(x + e, u);
                 load_unit<T, VEC>(dy + e, g);
                 float s1 = 0.f, s2 = 0.f;
#pragma unroll
                 for (int i = 0; i < VEC; ++i) { s1 += g[i]; s2 += g[i] * (u[i] - sh); }
                 a1 += s1; a2 += s2;
               },
               [&](long long e) { const float g = to_f<T>(dy[e]); a1 += g; a2 += g * (to_f<T>(x[e]) - sh); });
  } else {
    visit<VEC>(f, B, F, R, sp,
               [&](long long e) {
                 float u[VEC];
                 load_unit<T, VEC>(x + e, u);
                 float s1 = 0.f, s2 = 0.f;
#pragma unroll
                 for (int i = 0; i < VEC; ++i) { const float v = u[i] - sh; s1 += v; s2 += v * v; }
                 a1 += s1; a2 += s2;
               },
               [&](long long e) { const float v = to_f<T>(x[e]) - sh; a1 += v; a2 += v * v; });
  }
  a1 = block_sum_bn(a1, red);
  if (mode != 0) a2 = block_sum_bn(a2, red);
  if (threadIdx.x == 0) {
    if (PARTIALS) {
      float* o = out + ((long long)f * gridDim.y + blockIdx.y) * 2;
      o[0] = a1; o[1] = a2;
    } else {
      atomicAdd(out + f, a1);
      if (mode != 0 && out2 != nullptr) atomicAdd(out2 + f, a2);
    }
  }
}

// Mean and sum of squared deviations of the union of two samples (Chan, Golub, LeVeque 1979).
struct Moments {
  float n, mean, m2;
};
__device__ __forceinline__ void merge(Moments& a, float n, float mean, float m2) {
  if (n <= 0.f) return;
  const float t = a.n + n, d = mean - a.mean, w = n / t;
  a.mean += d * w;
  a.m2 += m2 + d * w * a.n * d;                           // (no square that overflows where it counts for nothing)
  a.n = t;
}
__device__ __forceinline__ Moments warp_merge(Moments m) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float n = __shfl_xor_sync(0xffffffffu, m.n, o), mean = __shfl_xor_sync(0xffffffffu, m.mean, o),
                m2 = __shfl_xor_sync(0xffffffffu, m.m2, o);
    merge(m, n, mean, m2);
  }
  return m;
}

// One read of x instead of two (sum, then squared deviations from the mean): a unit's own mean and squared
// deviations are formed in registers and merged, which cancels no worse than the two-pass form.
// part[(f * gridDim.y + split) * 3] = {count, mean, M2}.
template <typename T, int VEC>
__global__ void __launch_bounds__(kBnThreads)
bn_moments_kernel(const T* __restrict__ x, int B, int F, long long R, Split sp, float* __restrict__ part) {
  __shared__ float red[3][kBnThreads / 32];
  Moments m{0.f, 0.f, 0.f};
  visit<VEC>(blockIdx.x, B, F, R, sp,
             [&](long long e) {
               float u[VEC];
               load_unit<T, VEC>(x + e, u);
               float s = 0.f, q = 0.f;
#pragma unroll
               for (int i = 0; i < VEC; ++i) s += u[i];
               s *= 1.f / VEC;
#pragma unroll
               for (int i = 0; i < VEC; ++i) { const float d = u[i] - s; q += d * d; }
               merge(m, (float)VEC, s, q);
             },
             [&](long long e) { merge(m, 1.f, to_f<T>(x[e]), 0.f); });
  m = warp_merge(m);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { red[0][warp] = m.n; red[1][warp] = m.mean; red[2][warp] = m.m2; }
  __syncthreads();
  if (warp == 0) {
    m = Moments{0.f, 0.f, 0.f};
    if (lane < kBnThreads / 32) m = Moments{red[0][lane], red[1][lane], red[2][lane]};
    m = warp_merge(m);
    if (lane == 0) {
      float* o = part + ((long long)blockIdx.x * gridDim.y + blockIdx.y) * 3;
      o[0] = m.n; o[1] = m.mean; o[2] = m.m2;
    }
  }
}

// One warp per feature: statistics of the batch, running statistics.  stat = [mean | rstd | sum (x - mean) | gamma] x F
// (gamma as it is now: it may change before the backward pass).
// Sums, mean and variance take the type of x on their way, as they do where they travel between workers: the
// results (and which of two equal values a following max pooling picks) do not depend on the number of workers.
// The gradient kernels below round in the same places.
__global__ void bn_moments_final_kernel(const float* __restrict__ part, int splits, int F, float count, float eps,
                                        float* __restrict__ stat, int dtype, const void* gamma, int gamma_dtype,
                                        void* run_mean, void* run_var,
                                        int run_dtype, float momentum, float unbias) {
  const int f = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (f >= F) return;
  Moments m{0.f, 0.f, 0.f};
  for (int s = lane; s < splits; s += 32) {
    const float* p = part + ((long long)f * splits + s) * 3;
    merge(m, p[0], p[1], p[2]);
  }
  m = warp_merge(m);
  if (lane) return;
  const float mean = dtype == 0 ? round_as(round_as(m.mean * count, 0) / count, 0) : m.mean;
  const float off = m.mean - mean;
  const float var = round_as(round_as(m.m2 + count * off * off, dtype) / count, dtype);
  stat[f] = mean;
  stat[F + f] = 1.f / sqrtf(var + eps);
  stat[2 * F + f] = count * off;
  stat[3 * F + f] = gamma == nullptr ? 1.f : load_as(gamma, gamma_dtype, f);
  if (run_mean != nullptr) {
    const float keep = 1.f - momentum;
    store_as(run_mean, run_dtype, f, round_as(keep * load_as(run_mean, run_dtype, f), run_dtype) +
                                         round_as(momentum * mean, dtype));
    store_as(run_var, run_dtype, f, round_as(keep * load_as(run_var, run_dtype, f), run_dtype) +
                                        round_as(momentum * round_as(var * unbias, dtype), dtype));
  }
}

// One warp per feature: coef = [a | b | c] x F of dx = a dy + b (x - mean) + c (through the normalisation, the
// squared deviations and the sum), and the parameter gradients.
__global__ void bn_grad_final_kernel(const float* __restrict__ part, int splits, int F, float count,
                                     const float* __restrict__ stat, int dtype, int gamma_dtype,
                                     float* __restrict__ coef, void* dgamma, void* dbeta, int beta_dtype) {
  const int f = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (f >= F) return;
  float s1 = 0.f, s2 = 0.f;
  for (int s = lane; s < splits; s += 32) {
    const float* p = part + ((long long)f * splits + s) * 2;
    s1 += p[0]; s2 += p[1];
  }
  s1 = warp_sum(s1); s2 = warp_sum(s2);
  if (lane) return;
  const float rstd = stat[F + f], g = stat[3 * F + f];
  const float a = g * rstd;
  const float dv = round_as(round_as(-0.5f * g * rstd * rstd * rstd * s2, dtype) / count, dtype);
  const float dmean = round_as(round_as(-a * s1, dtype) + round_as(-2.f * dv * stat[2 * F + f], dtype), dtype);
  coef[f] = a;
  coef[F + f] = 2.f * dv;
  coef[2 * F + f] = round_as(dmean / count, dtype);
  if (dgamma != nullptr) store_as(dgamma, gamma_dtype, f, rstd * s2);
  if (dbeta != nullptr) store_as(dbeta, beta_dtype, f, s1);
}

// Per-feature coefficients of  y = a (x - m) + c (+ e z):  given (kAffine), gamma * rstd, mean, beta from the batch
// statistics (kNormalize), or given, the terms rounded to T one by one and added in the order e z, a (x - m), c
// (kGradient).
enum MapMode { kAffine, kNormalize, kGradient };
struct Coef {
  const float *a, *m, *c, *e;
  const void *gamma, *beta;
  int gamma_dtype, beta_dtype;
};

// blockIdx.x walks the units of a plane (one more than fit, since a plane need not start on the grid),
// blockIdx.y the planes.
template <typename T, MapMode MODE>
__device__ __forceinline__ float map_value(float x, float z, bool has_z, float a, float m, float c, float ez) {
  if (MODE == kGradient) {
    constexpr int dt = sizeof(T) == 2 ? 0 : 1;
    return round_as(round_as(ez * z, dt) + round_as(a * (x - m), dt), dt) + c;
  }
  float v = a * (x - m) + c;
  if (has_z) v += ez * z;
  return v;
}
template <typename T, int VEC, MapMode MODE>
__global__ void __launch_bounds__(kBnThreads)
bn_map_kernel(const T* __restrict__ x, const T* __restrict__ z, const Coef k, int F, int planes, long long R,
              T* __restrict__ y) {
  const long long pos = blockIdx.x * (long long)blockDim.x + threadIdx.x;
#pragma unroll 2
  for (int pl = blockIdx.y; pl < planes; pl += gridDim.y) {
    const int f = pl % F;
    const long long p0 = pl * R, p1 = p0 + R, e = (p0 / VEC + pos) * VEC;
    if (e >= p1) continue;
    float a = k.a[f];
    const float m = k.m ? k.m[f] : 0.f;
    float c = 0.f;
    if (MODE == kNormalize) {
      if (k.gamma != nullptr) a *= load_as(k.gamma, k.gamma_dtype, f);
      if (k.beta != nullptr) c = load_as(k.beta, k.beta_dtype, f);
    } else if (k.c) {
      c = k.c[f];
    }
    const float ez = z != nullptr ? k.e[f] : 0.f;
    if (VEC == 1 || (e >= p0 && e + VEC <= p1)) {
      float v[VEC], w[VEC];
      load_unit<T, VEC>(x + e, v);
      if (z != nullptr) load_unit<T, VEC>(z + e, w);
#pragma unroll
      for (int i = 0; i < VEC; ++i) v[i] = map_value<T, MODE>(v[i], w[i], z != nullptr, a, m, c, ez);
      store_unit<T, VEC>(y + e, v);
    } else {
      for (int i = 0; i < VEC; ++i)
        if (e + i >= p0 && e + i < p1) {
          const float w = z != nullptr ? to_f<T>(z[e + i]) : 0.f;
          y[e + i] = from_f<T>(map_value<T, MODE>(to_f<T>(x[e + i]), w, z != nullptr, a, m, c, ez));
        }
    }
  }
}

Split split_for(int B, int F, long long R, int vec) {
  Split sp;
  const long long nu = (R + vec - 1) / vec + (vec > 1 ? 1 : 0);
  sp.tpb = 1;
  while (sp.tpb < kBnThreads && sp.tpb < nu) sp.tpb *= 2;
  const int rows = kBnThreads / sp.tpb;
  const long long want = (148 * 8 + F - 1) / F;          // enough CTAs to fill the GPU
  long long su = (nu + sp.tpb * 4LL - 1) / (sp.tpb * 4LL);
  if (su > want) su = want;
  if (su > 2048) su = 2048;
  long long sb = (B + rows - 1) / rows;
  if (sb > want / su) sb = want / su;
  if (sb < 1) sb = 1;
  if (sb > 31) sb = 31;                                   // su * sb stays below the grid's limit
  sp.su = (int)su; sp.sb = (int)sb;
  return sp;
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <typename T, MapMode MODE>
int map(const T* x, const T* z, const Coef& k, int B, int F, long long R, T* y, cudaStream_t s) {
  constexpr int V = 16 / sizeof(T);
  const bool vec = aligned16(x) && aligned16(y) && (z == nullptr || aligned16(z));
  const long long units = vec ? (R + V - 1) / V + 1 : R;
  const long long planes = (long long)B * F;
  if (planes > 0x7fffffffLL) return DD_ERR_TOO_LARGE;
  const int t = units >= kBnThreads ? kBnThreads : (int)((units + 31) / 32 * 32);
  const long long bx = (units + t - 1) / t;
  long long by = (148LL * 32 + bx - 1) / bx;
  if (by > planes) by = planes;
  if (by > 65535) by = 65535;
  const dim3 grid((unsigned)bx, (unsigned)by);
  if (vec) bn_map_kernel<T, V, MODE><<<grid, t, 0, s>>>(x, z, k, F, (int)planes, R, y);
  else     bn_map_kernel<T, 1, MODE><<<grid, t, 0, s>>>(x, z, k, F, (int)planes, R, y);
  return (int)cudaGetLastError();
}

template <typename T, bool PARTIALS>
int reduce(const T* x, const T* dy, const float* shift, int B, int F, long long R, int mode, const Split& sp, bool vec,
           float* out, float* out2, cudaStream_t s) {
  const dim3 grid((unsigned)F, (unsigned)(sp.su * sp.sb));
  if (vec)
    bn_reduce_kernel<T, 16 / sizeof(T), PARTIALS><<<grid, kBnThreads, 0, s>>>(x, dy, shift, B, F, R, mode, sp, out, out2);
  else
    bn_reduce_kernel<T, 1, PARTIALS><<<grid, kBnThreads, 0, s>>>(x, dy, shift, B, F, R, mode, sp, out, out2);
  return (int)cudaGetLastError();
}

template <typename T>
int train_fwd(const T* x, const void* gamma, const void* beta, int gamma_dtype, int beta_dtype, int B, int F, long long R,
              float eps, void* run_mean, void* run_var, int run_dtype, float momentum, float* ws, float* stat, T* y,
              cudaStream_t s) {
  constexpr int V = 16 / sizeof(T);
  const bool vec = aligned16(x);
  const Split sp = split_for(B, F, R, vec ? V : 1);
  const int splits = sp.su * sp.sb;
  const dim3 grid((unsigned)F, (unsigned)splits);
  if (vec) bn_moments_kernel<T, V><<<grid, kBnThreads, 0, s>>>(x, B, F, R, sp, ws);
  else     bn_moments_kernel<T, 1><<<grid, kBnThreads, 0, s>>>(x, B, F, R, sp, ws);
  const double n = (double)B * (double)R;
  bn_moments_final_kernel<<<(F + 7) / 8, 256, 0, s>>>(ws, splits, F, (float)n, eps, stat,
                                                      sizeof(T) == 2 ? 0 : 1, gamma, gamma_dtype, run_mean, run_var,
                                                      run_dtype, momentum,
                                                      (float)(n / (n - 1.0 > 1.0 ? n - 1.0 : 1.0)));
  Coef k{stat + F, stat, nullptr, nullptr, gamma, beta, gamma_dtype, beta_dtype};
  return map<T, kNormalize>(x, nullptr, k, B, F, R, y, s);
}

template <typename T>
int train_bwd(const T* x, const T* dy, int gamma_dtype, int beta_dtype, int B, int F, long long R, const float* stat,
              float* ws, float* coef, T* dx, void* dgamma, void* dbeta, cudaStream_t s) {
  const bool vec = aligned16(x) && aligned16(dy);
  const Split sp = split_for(B, F, R, vec ? 16 / (int)sizeof(T) : 1);
  int r = reduce<T, true>(x, dy, stat, B, F, R, 2, sp, vec, ws, nullptr, s);
  if (r) return r;
  bn_grad_final_kernel<<<(F + 7) / 8, 256, 0, s>>>(ws, sp.su * sp.sb, F, (float)((double)B * (double)R), stat,
                                                   sizeof(T) == 2 ? 0 : 1, gamma_dtype, coef, dgamma, dbeta, beta_dtype);
  if (dx == nullptr) return (int)cudaGetLastError();
  // dx = a dy + b (x - mean) + c
  Coef k{coef + F, stat, coef + 2 * F, coef, nullptr, nullptr, 1, 1};
  return map<T, kGradient>(x, dy, k, B, F, R, dx, s);
}

}  // namespace

// dtype: 0 = bf16, 1 = fp32.  x (and dy in mode 2): [B, F, R] contiguous; shift: [F] fp32 or null;
// out / out2: [F] fp32, zero on entry.
DD_API int dd_bn_reduce(const void* x, const void* dy, const float* shift, int B, int F, long long R, int mode,
                        int dtype, float* out, float* out2, void* stream) {
  if (B <= 0 || F <= 0 || R <= 0 || mode < 0 || mode > 2 || out == nullptr) return DD_ERR_BAD_ARG;
  if (mode == 2 && dy == nullptr) return DD_ERR_BAD_ARG;
  const bool vec = aligned16(x) && (mode != 2 || aligned16(dy));
  const Split sp = split_for(B, F, R, !vec ? 1 : dtype == 0 ? 8 : 4);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (dtype == 0)
    return reduce<__nv_bfloat16, false>(reinterpret_cast<const __nv_bfloat16*>(x),
                                        reinterpret_cast<const __nv_bfloat16*>(dy), shift, B, F, R, mode, sp, vec, out,
                                        out2, s);
  return reduce<float, false>(reinterpret_cast<const float*>(x), reinterpret_cast<const float*>(dy), shift, B, F, R, mode,
                              sp, vec, out, out2, s);
}

// y = a[f] * (x - m[f]) + c[f] (+ e[f] * z); m, c may be null (0); z / e null together.
DD_API int dd_bn_affine(const void* x, const void* z, const float* a, const float* m, const float* c, const float* e,
                        int B, int F, long long R, int dtype, void* y, void* stream) {
  if (B <= 0 || F <= 0 || R <= 0 || a == nullptr || (z != nullptr) != (e != nullptr)) return DD_ERR_BAD_ARG;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  Coef k{a, m, c, e, nullptr, nullptr, 1, 1};
  if (dtype == 0)
    return map<__nv_bfloat16, kAffine>(reinterpret_cast<const __nv_bfloat16*>(x), reinterpret_cast<const __nv_bfloat16*>(z),
                              k, B, F, R, reinterpret_cast<__nv_bfloat16*>(y), s);
  return map<float, kAffine>(reinterpret_cast<const float*>(x), reinterpret_cast<const float*>(z), k, B, F, R,
                    reinterpret_cast<float*>(y), s);
}

// Floats of workspace that dd_bn_train_fwd / _bwd need (an upper bound for either type).
DD_API int dd_bn_train_workspace(int B, int F, long long R) {
  if (B <= 0 || F <= 0 || R <= 0) return 0;
  int most = 0;
  for (int vec : {1, 4, 8}) {
    const Split sp = split_for(B, F, R, vec);
    if (sp.su * sp.sb > most) most = sp.su * sp.sb;
  }
  return 3 * most * F;
}

// Batch norm of one worker's whole batch.  stat: [4, F] fp32 (mean, 1 / sqrt(var + eps), sum (x - mean), gamma), kept
// for the backward pass; gamma / beta / run_*: [F] in their own types (0 = bf16, 1 = fp32) or null.
DD_API int dd_bn_train_fwd(const void* x, const void* gamma, const void* beta, int gamma_dtype, int beta_dtype, int B,
                           int F, long long R, int dtype, float eps, void* run_mean, void* run_var, int run_dtype,
                           float momentum, float* ws, float* stat, void* y, void* stream) {
  if (B <= 0 || F <= 0 || R <= 0 || ws == nullptr || stat == nullptr || (run_mean == nullptr) != (run_var == nullptr))
    return DD_ERR_BAD_ARG;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (dtype == 0)
    return train_fwd<__nv_bfloat16>(reinterpret_cast<const __nv_bfloat16*>(x), gamma, beta, gamma_dtype, beta_dtype, B, F,
                                    R, eps, run_mean, run_var, run_dtype, momentum, ws, stat,
                                    reinterpret_cast<__nv_bfloat16*>(y), s);
  return train_fwd<float>(reinterpret_cast<const float*>(x), gamma, beta, gamma_dtype, beta_dtype, B, F, R, eps, run_mean,
                          run_var, run_dtype, momentum, ws, stat, reinterpret_cast<float*>(y), s);
}

// coef: [3, F] fp32 scratch; dx, dgamma, dbeta may be null.
DD_API int dd_bn_train_bwd(const void* x, const void* dy, int gamma_dtype, int beta_dtype, int B, int F, long long R,
                           int dtype, const float* stat, float* ws, float* coef, void* dx, void* dgamma, void* dbeta,
                           void* stream) {
  if (B <= 0 || F <= 0 || R <= 0 || ws == nullptr || stat == nullptr || coef == nullptr) return DD_ERR_BAD_ARG;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (dtype == 0)
    return train_bwd<__nv_bfloat16>(reinterpret_cast<const __nv_bfloat16*>(x), reinterpret_cast<const __nv_bfloat16*>(dy),
                                    gamma_dtype, beta_dtype, B, F, R, stat, ws, coef,
                                    reinterpret_cast<__nv_bfloat16*>(dx), dgamma, dbeta, s);
  return train_bwd<float>(reinterpret_cast<const float*>(x), reinterpret_cast<const float*>(dy), gamma_dtype, beta_dtype,
                          B, F, R, stat, ws, coef, reinterpret_cast<float*>(dx), dgamma, dbeta, s);
}
