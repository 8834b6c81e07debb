// pdl.cuh -- programmatic dependent launch of the query path's kernels.
//
// The kernels of a query call form a chain (projection, location, order or
// head, search), and for small batches the gaps between them are a fifth of
// the call.  A kernel launched with launch_pdl may be set up while its
// predecessor in the stream still runs.  It therefore begins with
// dependency_wait(), before it reads or writes anything: that returns once
// every kernel before it has completed and its writes are visible.
// allow_dependents() lets the successor's set-up start; it only concerns that
// successor's launch, whose own wait still covers this whole kernel.
#pragma once
#include <cuda_runtime.h>

namespace rte {

__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Batches that the early set-up pays for: small ones, and graph replays, whose
// live size is read on the device.  On one GB300: one query 134 -> 129 us, 37
// learned queries 97.5 -> 93.4 us, uneven batches through the graph 2039 ->
// 2014 us; but 10k learned queries 490 -> 513 us, as the head's CTAs then take
// their SMs before the kernels on the side stream do.
constexpr long long kPdlRows = 4096;

inline cudaError_t launch_pdl(const void* kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t st, void** args,
                              long long rows, const void* rows_dev) {
  if (!rows_dev && rows > kPdlRows) return cudaLaunchKernel(kernel, grid, block, args, smem, st);
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelExC(&cfg, kernel, args);
}

}  // namespace rte
