// gw_launch.h -- dependent launches: a kernel whose launch, prologue and first
// loads of constant data overlap the kernel before it in the stream.
//
// A kernel launched with launch_dependent may start once every block of the
// kernel before it has called dep_launch() or exited.  It calls dep_wait()
// before its first access to anything an earlier kernel of the stream writes
// or reads: that wait ends when the kernel before it has completed and its
// writes are visible.  Every kernel of such a chain waits, so all earlier
// kernels have completed too.  After a copy or an event in the stream the
// launch is an ordinary one.
//
// What such a kernel reads changes while it is resident, so of its parameters
// only arrays that no kernel of the chain writes are __restrict__: of the others
// the compiler could move loads above the wait, or read them by the path that
// takes data to be unchanged for the whole kernel.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace gw {

#ifdef __CUDACC__
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

template <typename... P, typename... A>
cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);
}

}  // namespace gw
