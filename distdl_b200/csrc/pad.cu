// Shifted copy of the spatial dimensions of [planes, n0, n1, n2] tensors (contiguous, 2- or 4-byte elements):
//
//   dst[p, o] = src[p, o - lo]   where that lies inside src, else `fill`
//
// With lo >= 0 and a larger dst this is the zero (or -inf) padding in front of a convolution or a pooling layer,
// with lo <= 0 and a smaller dst the crop that is its adjoint.  Stands where the reference calls
// torch.nn.functional.pad (src/distdl/nn/conv_feature.py, pooling.py).
//
// Bound by memory.  A thread fixes V neighbours of one row of dst (16 bytes where the row's length allows it), so
// that stores are wide whatever the shift does to the loads, and walks the planes; the loads, which start at any
// element, are single and meet in L1.  [8, 64, 256, 256] bf16 by one on every side: 31 us (fill and strided
// copy: 98), the crop 26 us (strided copy: 81).
#include "common.cuh"
#include "runtime.cuh"

namespace {

struct ShiftGeom {
  int in[3], out[3], lo[3];
  long long planes;
};

template <typename W, int V> struct Pack;
template <> struct Pack<uint16_t, 8> { using type = uint4; };
template <> struct Pack<uint16_t, 4> { using type = uint2; };
template <> struct Pack<uint16_t, 2> { using type = uint32_t; };
template <> struct Pack<uint16_t, 1> { using type = uint16_t; };
template <> struct Pack<uint32_t, 4> { using type = uint4; };
template <> struct Pack<uint32_t, 2> { using type = uint2; };
template <> struct Pack<uint32_t, 1> { using type = uint32_t; };

template <typename W, int V>
__global__ void __launch_bounds__(256)
shift_copy_kernel(const W* __restrict__ src, W* __restrict__ dst, const ShiftGeom g, W fill) {
  using P = typename Pack<W, V>::type;
  const long long out_plane = (long long)g.out[0] * g.out[1] * g.out[2];
  const long long in_plane = (long long)g.in[0] * g.in[1] * g.in[2];
  const long long first = (blockIdx.x * (long long)blockDim.x + threadIdx.x) * V;
  if (first >= out_plane) return;
  long long r = first;
  const int o2 = (int)(r % g.out[2]); r /= g.out[2];
  const int i1 = (int)(r % g.out[1]) - g.lo[1], i0 = (int)(r / g.out[1]) - g.lo[0], i2 = o2 - g.lo[2];
  const bool row = i0 >= 0 && i0 < g.in[0] && i1 >= 0 && i1 < g.in[1];
  const long long off = ((long long)i0 * g.in[1] + i1) * g.in[2] + i2;
  bool live[V];
#pragma unroll
  for (int v = 0; v < V; ++v) live[v] = row && i2 + v >= 0 && i2 + v < g.in[2];
  const W* s = src + blockIdx.y * in_plane + off;
  W* d = dst + blockIdx.y * out_plane + first;
  const long long sstep = gridDim.y * in_plane, dstep = gridDim.y * out_plane;
#pragma unroll (V >= 4 ? 2 : 4)
  for (int left = (int)((g.planes - blockIdx.y + gridDim.y - 1) / gridDim.y); left > 0; --left, s += sstep, d += dstep) {
    union { W w[V]; P pack; } u;
#pragma unroll
    for (int v = 0; v < V; ++v) u.w[v] = live[v] ? __ldg(s + v) : fill;
    *reinterpret_cast<P*>(d) = u.pack;
  }
}

template <typename W, int V>
int launch(const void* src, void* dst, const ShiftGeom& g, W fill, cudaStream_t s) {
  const long long n = (long long)g.out[0] * g.out[1] * g.out[2] / V;
  const int t = n >= 256 ? 256 : (int)((n + 31) / 32 * 32);
  const long long bx = (n + t - 1) / t;
  long long by = (148LL * 16 + bx - 1) / bx;             // about sixteen CTAs per SM in all
  if (by > g.planes) by = g.planes;
  if (by > 65535) by = 65535;
  shift_copy_kernel<W, V><<<dim3((unsigned)bx, (unsigned)by), t, 0, s>>>(reinterpret_cast<const W*>(src),
                                                                         reinterpret_cast<W*>(dst), g, fill);
  return (int)cudaGetLastError();
}

template <typename W>
int run(const void* src, void* dst, const ShiftGeom& g, W fill, cudaStream_t s) {
  // rows of dst start on V elements when their length is a multiple of V and dst starts on 16 bytes
  const bool aligned = (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
  if constexpr (sizeof(W) == 2)
    if (aligned && g.out[2] % 8 == 0) return launch<W, 8>(src, dst, g, fill, s);
  if (aligned && g.out[2] % 4 == 0) return launch<W, 4>(src, dst, g, fill, s);
  if (aligned && g.out[2] % 2 == 0) return launch<W, 2>(src, dst, g, fill, s);
  return launch<W, 1>(src, dst, g, fill, s);
}

// ------------------------------------------------------------------ between channels-first and channels-last
// The same shifted copy into or out of the layout [batch, n0, n1, n2, C] that the tensor-core convolutions work in,
// so that padding, crop and change of layout are one pass, for 2-byte elements.  A CTA moves 2048 words (pairs of channels)
// through shared memory, W of each position: channels-first side consecutive positions, channels-last side 16 bytes per
// thread, both without bank conflicts.  W follows the channels, because a CTA for 64 of them is idle where there are 8, and
// positions are decoded in 32 bits where a plane allows it.  bf16, padded by one, us, to channels-last | back, 32 words and 64
// bits -> now: [8, 64, 256, 256] 51 | 35 -> 51 | 33, [6, 8, 87^3] 131 | 187 -> 49 | 29, [8, 16, 300, 300] 27 | 37 -> 12 | 12, [4, 24, 60^3]
// 41 | 47 -> 25 | 25 (the library's own conversion inside the convolution at the first size: 64 | 46 behind 31 | 26 for padding
// and crop).
template <int W>
struct ChannelTile {
  static constexpr int POS = 2048 / W;                       // positions
  static constexpr int PITCH = POS + (W == 32 ? 1 : W == 16 ? 2 : W == 8 ? 4 : 0);
  static constexpr int PER = POS > 256 ? POS / 256 : 1;      // positions of a thread on the channels-first side
  static constexpr int STEP = POS > 256 ? 1 : 256 / POS;     // distance of its words there
};

// the pair of channels at p, zero outside
__device__ __forceinline__ uint32_t gather_pair(const uint16_t* p, long long step, bool live) {
  const uint32_t a = live ? __ldg(p) : 0, b = live ? __ldg(p + step) : 0;
  return a | (b << 16);
}

// position of dst -> offset (in positions) inside a plane of src, -1 outside.  I: unsigned where a plane has fewer than 2^31.
template <typename I>
__device__ __forceinline__ long long source_position(const ShiftGeom& g, I o) {
  const I row = o / (I)g.out[2], sheet = row / (I)g.out[1];
  const int i2 = (int)(o - row * (I)g.out[2]) - g.lo[2];
  const int i1 = (int)(row - sheet * (I)g.out[1]) - g.lo[1], i0 = (int)sheet - g.lo[0];
  const bool live = i0 >= 0 && i0 < g.in[0] && i1 >= 0 && i1 < g.in[1] && i2 >= 0 && i2 < g.in[2];
  return live ? ((long long)i0 * g.in[1] + i1) * g.in[2] + i2 : -1;
}

template <int W, typename I>
__global__ void __launch_bounds__(256)
to_channels_last_kernel(const uint16_t* __restrict__ src, uint16_t* __restrict__ dst, const ShiftGeom g, int C) {
  using T = ChannelTile<W>;
  __shared__ uint32_t tile[W][T::PITCH];
  const long long out_plane = (long long)g.out[0] * g.out[1] * g.out[2];
  const long long in_plane = (long long)g.in[0] * g.in[1] * g.in[2];
  const long long p0 = blockIdx.x * (long long)T::POS;
  const int c0 = blockIdx.y * W * 2, w0 = T::POS > 256 ? 0 : threadIdx.x / T::POS;
#pragma unroll
  for (int k = 0; k < T::PER; ++k) {
    const int pos = (threadIdx.x & (T::POS - 1)) + 256 * k;
    const long long at = p0 + pos < out_plane ? source_position<I>(g, (I)(p0 + pos)) : -1;
    const uint16_t* s = src + ((long long)blockIdx.z * C + c0 + w0 * 2) * in_plane + (at < 0 ? 0 : at);
#pragma unroll
    for (int w = w0; w < W; w += T::STEP) {
      if (c0 + w * 2 < C) tile[w][pos] = gather_pair(s, in_plane, at >= 0);
      s += T::STEP * 2 * in_plane;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int idx = threadIdx.x + 256 * k, chunk = idx & (W / 4 - 1), pos = idx / (W / 4), c = c0 + chunk * 8;
    if (c >= C || p0 + pos >= out_plane) continue;
    const uint4 v = make_uint4(tile[chunk * 4][pos], tile[chunk * 4 + 1][pos], tile[chunk * 4 + 2][pos],
                               tile[chunk * 4 + 3][pos]);
    *reinterpret_cast<uint4*>(dst + ((long long)blockIdx.z * out_plane + p0 + pos) * C + c) = v;
  }
}

template <int W, typename I>
__global__ void __launch_bounds__(256)
from_channels_last_kernel(const uint16_t* __restrict__ src, uint16_t* __restrict__ dst, const ShiftGeom g, int C) {
  using T = ChannelTile<W>;
  __shared__ uint32_t tile[W][T::PITCH];
  const long long out_plane = (long long)g.out[0] * g.out[1] * g.out[2];
  const long long in_plane = (long long)g.in[0] * g.in[1] * g.in[2];
  const long long p0 = blockIdx.x * (long long)T::POS;
  const int c0 = blockIdx.y * W * 2;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int idx = threadIdx.x + 256 * k, chunk = idx & (W / 4 - 1), pos = idx / (W / 4), c = c0 + chunk * 8;
    if (c >= C || p0 + pos >= out_plane) continue;
    const long long at = source_position<I>(g, (I)(p0 + pos));
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (at >= 0) v = __ldg(reinterpret_cast<const uint4*>(src + ((long long)blockIdx.z * in_plane + at) * C + c));
    tile[chunk * 4][pos] = v.x; tile[chunk * 4 + 1][pos] = v.y;
    tile[chunk * 4 + 2][pos] = v.z; tile[chunk * 4 + 3][pos] = v.w;
  }
  __syncthreads();
  const int w0 = T::POS > 256 ? 0 : threadIdx.x / T::POS;
#pragma unroll
  for (int k = 0; k < T::PER; ++k) {
    const int pos = (threadIdx.x & (T::POS - 1)) + 256 * k;
    if (p0 + pos >= out_plane) return;
    uint16_t* d = dst + ((long long)blockIdx.z * C + c0 + w0 * 2) * out_plane + p0 + pos;
#pragma unroll
    for (int w = w0; w < W; w += T::STEP) {
      if (c0 + w * 2 < C) {
        const uint32_t v = tile[w][pos];
        d[0] = (uint16_t)v;
        d[out_plane] = (uint16_t)(v >> 16);
      }
      d += T::STEP * 2 * out_plane;
    }
  }
}

// Words of a position that a CTA takes: as many as leave no more than a fifth of the threads without channels; 32 bytes or
// more, a sector.  Into channels-last memory 32 of them where there are too few CTAs to fill the SMs ten times: each has fewer
// positions to decode then, and idle threads cost nothing.  us, 32 words -> fewer: [1, 8, 80^2] 2.3 -> 3.5, [8, 8, 80^2] 3.3 -> 3.7, [4, 24,
// 120^2] 4.1 -> 4.1; [8, 8, 120^2] 5.3 -> 3.9, [4, 24, 160^2] 5.7 -> 5.1.  Back it makes no difference (2.5 -> 2.3 for the first).
int channel_words(int to_last, int B, int C, long long positions) {
  auto fits = [C](int w) { return (C + w * 2 - 1) / (w * 2) * (w * 2) * 4 <= C * 5; };
  if (to_last && (positions + 63) / 64 * ((C + 63) / 64) * B < 10LL * dd::current_sm_count()) return 32;
  return C <= 8 ? 4 : fits(32) ? 32 : fits(16) ? 16 : 8;
}

template <int W>
int launch_channels(const uint16_t* src, uint16_t* dst, int to_last, int B, int C, const ShiftGeom& g, cudaStream_t s) {
  const long long n = (long long)g.out[0] * g.out[1] * g.out[2];
  const dim3 grid((unsigned)((n + ChannelTile<W>::POS - 1) / ChannelTile<W>::POS), (unsigned)((C + W * 2 - 1) / (W * 2)),
                  (unsigned)B);
  const bool small = n < 0x7fffffffLL;
  auto kernel = to_last ? (small ? to_channels_last_kernel<W, unsigned> : to_channels_last_kernel<W, long long>)
                        : (small ? from_channels_last_kernel<W, unsigned> : from_channels_last_kernel<W, long long>);
  kernel<<<grid, 256, 0, s>>>(src, dst, g, C);
  return (int)cudaGetLastError();
}

}  // namespace

// esize: bytes per element (2 or 4); fill: the element's bits (low esize bytes).
DD_API int dd_shift_copy(const void* src, void* dst, int esize, long long planes, const int* in, const int* out,
                         const int* lo, unsigned fill, void* stream) {
  if (src == nullptr || dst == nullptr || planes <= 0 || (esize != 2 && esize != 4)) return DD_ERR_BAD_ARG;
  ShiftGeom g;
  g.planes = planes;
  for (int i = 0; i < 3; ++i) {
    if (in[i] <= 0 || out[i] <= 0) return DD_ERR_BAD_ARG;
    g.in[i] = in[i]; g.out[i] = out[i]; g.lo[i] = lo[i];
  }
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return esize == 2 ? run<uint16_t>(src, dst, g, (uint16_t)fill, s) : run<uint32_t>(src, dst, g, fill, s);
}

// The same between [B, C, in...] and [B, out..., C] (to_last = 1) or [B, in..., C] and [B, C, out...] (to_last = 0) of
// 2-byte elements, filled with zeros.  C: a multiple of 8; the channels-last tensor 16-byte aligned.
DD_API int dd_shift_channels(const void* src, void* dst, int to_last, int B, int C, const int* in, const int* out,
                             const int* lo, void* stream) {
  if (src == nullptr || dst == nullptr || B <= 0 || B > 65535 || C <= 0 || C % 8) return DD_ERR_BAD_ARG;
  if (reinterpret_cast<uintptr_t>(to_last ? dst : src) & 15) return DD_ERR_ALIGN;
  ShiftGeom g;
  g.planes = 0;
  for (int i = 0; i < 3; ++i) {
    if (in[i] <= 0 || out[i] <= 0) return DD_ERR_BAD_ARG;
    g.in[i] = in[i]; g.out[i] = out[i]; g.lo[i] = lo[i];
  }
  const uint16_t* from = reinterpret_cast<const uint16_t*>(src);
  uint16_t* to = reinterpret_cast<uint16_t*>(dst);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const int words = channel_words(to_last, B, C, (long long)g.out[0] * g.out[1] * g.out[2]);
  if (words == 4) return launch_channels<4>(from, to, to_last, B, C, g, st);
  if (words == 8) return launch_channels<8>(from, to, to_last, B, C, g, st);
  if (words == 16) return launch_channels<16>(from, to, to_last, B, C, g, st);
  return launch_channels<32>(from, to, to_last, B, C, g, st);
}

// The words of a position that a CTA takes in the call above, for tests.
DD_API int dd_shift_channels_words(int to_last, int B, int C, long long positions) {
  return channel_words(to_last, B, C, positions);
}
