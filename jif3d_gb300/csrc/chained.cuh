// chained.cuh -- launches whose start overlaps the end of the kernel before
// them in the stream (programmatic dependent launch).
//
// An evaluation of a small survey is a handful of kernels of one to ten
// microseconds, each waiting for the one before.  A kernel launched by
// launch_chained may get its blocks onto the SMs while the kernel before it
// still runs, as soon as that one has called chain_begin() in every block (a
// kernel that never calls it counts at its end); chain_wait() then waits until
// the kernel before has finished and its writes are visible.  Every chained
// kernel calls chain_wait() before it reads or writes memory that any other
// kernel touches, so that each finished kernel stands for all those before it.
#pragma once
#include <cuda_runtime.h>

namespace j3g {

__device__ __forceinline__ void chain_begin() { cudaTriggerProgrammaticLaunchCompletion(); }
__device__ __forceinline__ void chain_wait() { cudaGridDependencySynchronize(); }

template <class... P, class... A>
inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, int threads, size_t smem,
                                  cudaStream_t st, const A &...args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, P(args)...);
  if (e != cudaSuccess) cudaGetLastError();  // returned here, not by the next launch's check
  return e;
}

}  // namespace j3g
