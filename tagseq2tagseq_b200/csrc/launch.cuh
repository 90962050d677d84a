// Launches that may start before the launch before them in the stream has ended.
//
// A kernel of a chain is started while its predecessor still runs, sets itself up and waits in after_previous() for the
// predecessor's end; all of the predecessor's writes are visible then.  What the predecessor wrote is read with plain loads or
// bulk copies: a read-only load could be moved up across the wait.  The first kernel of a chain is an ordinary launch, which
// only calls let_next_start(), and every kernel after it waits in at least one thread of every block, so that a kernel's end
// implies the end of all before it.
#pragma once
#include <cuda_runtime.h>

namespace ts2ts {

__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void after_previous() {
  let_next_start();
  wait_previous();
}

// An ordinary launch unless `early`; the kernel's waits then find nothing to wait for.
template <typename... Params, typename... Args>
inline cudaError_t launch_after_if(bool early, void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = early;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}
template <typename... Params, typename... Args>
inline cudaError_t launch_after(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream, const Args&... args) {
  return launch_after_if(true, kernel, grid, threads, smem, stream, args...);
}

}  // namespace ts2ts
