// Host-side runtime shared by all entry points: per-device status record,
// driver entry points resolved at run time (no link-time libcuda dependency),
// tensor-map cache.
#pragma once

#include <cudaTypedefs.h>

#include "common.cuh"

namespace dd {

// Device pointer to this device's status record (allocated on first use).
StatusRecord* device_status(int* err);

// cuTensorMapEncodeTiled resolved through the runtime.
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder();

// Encodes (or fetches from a small cache) a rank-3 bf16 tensor map with a
// 128-byte swizzle: dims {inner, outer, batch}, strides in BYTES for outer
// and batch, box {box_inner, box_outer, 1}.  Returns 0 on success.
int get_tensor_map_bf16_3d(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer,
                           uint64_t batch, uint64_t outer_stride_bytes, uint64_t batch_stride_bytes,
                           uint32_t box_inner, uint32_t box_outer);

// The same for fp32 elements (outputs written or reduced by TMA).
int get_tensor_map_f32_3d(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer,
                          uint64_t batch, uint64_t outer_stride_bytes, uint64_t batch_stride_bytes,
                          uint32_t box_inner, uint32_t box_outer);

// A rank-4 bf16 tensor map of [rows, heads, D] tensors of several sequences: dims {inner, rows, heads, sequences}, box
// {box_inner, box_rows, 1, 1}.  Rows behind the end of a sequence read as zeros.
int get_tensor_map_bf16_4d(CUtensorMap* out, const void* base, uint64_t inner, uint64_t rows, uint64_t heads,
                           uint64_t sequences, uint64_t row_stride_bytes, uint64_t head_stride_bytes,
                           uint64_t sequence_stride_bytes, uint32_t box_inner, uint32_t box_rows);

int current_sm_count();

// Launches a kernel that calls grid_dependency_wait() before it touches global memory, so that its start (launch latency,
// barriers, tensor memory: 2 to 4 us) does not wait for the end of the kernel before it.  The products do so, and the kernels
// that mostly come before one let it start.  A training step of four layers of 1600 columns, 2 x 4096 tokens, 306 launches:
// 13 980 -> 13 720 us; four layers of 2048 columns, 3000 tokens: 7 180 -> 7 060.
// ahead: false for a kernel that leaves SMs to other streams, which would otherwise hold its SMs before it can work on them.
template <typename... P, typename... A>
inline int launch_ahead(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, bool ahead,
                        const A&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = ahead ? 1 : 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

}  // namespace dd
