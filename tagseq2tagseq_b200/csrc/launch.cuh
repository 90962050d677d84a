// Every kernel of this library is launched as one that need not find its predecessor in the stream ended: an ordinary launch
// behind another kernel starts at the next tick of a 2 us clock (B200, driver 580: 148 blocks that spin, back to back: 1.0 us a kernel 4.2 us apart
// and 2.3 us 6.2 apart; launched like this 2.2 and 3.4; inside a graph 2.2 and 3.4 either way).
//
// Unless the predecessor calls let_next_start() in all of its blocks, it has ended when such a kernel starts, but its writes need not be
// visible: that is what wait_previous() is for.  Where it does, the kernel sets itself up while the predecessor still runs and waits for its end there.
// A kernel touches no memory that another launch may have written or may still read before it has waited, and waits in at least one
// thread of every block, so that a kernel's end implies the end of all before it.  The first kernel of a chain (pre-pass, backward) calls let_next_start()
// behind its own wait: all that came before the chain has ended when its later kernels start, and these wait for what the chain itself has written.
// What may have been written just before is read with plain loads, bulk copies, through settled() or at addresses that come from such loads: another read-only load could be
// moved up across the wait.
#pragma once
#include <cuda_runtime.h>

namespace ts2ts {

__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// For a chain's inner kernels, whose predecessors trigger behind a wait of their own.
__device__ __forceinline__ void after_previous() {
  let_next_start();
  wait_previous();
}
// A pointer whose loads stay behind the wait that comes before, read-only ones too.
template <typename T> __device__ __forceinline__ T* settled(T* p) {
  asm volatile("" : "+l"(p)::"memory");
  __builtin_assume(p == nullptr || __isGlobal(p));
  return p;
}

template <typename... Params, typename... Args>
inline cudaError_t launch_after(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
  if (e != cudaSuccess) cudaGetLastError();  // the caller has it; the next launch's check must not find it
  return e;
}

}  // namespace ts2ts
