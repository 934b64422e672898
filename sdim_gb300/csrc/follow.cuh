// Launches that follow another kernel closely: the next kernel of a stream is
// set up while the one before it ends, instead of behind its end.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace sdim {

// First statement of a kernel that launch_following may launch: waits for the
// kernels before it on the stream to be complete, their writes visible (at once
// when it was launched in the ordinary way).
__device__ __forceinline__ void follow_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// In the kernel in front: the following one may take its place on the SMs from
// here on, once every CTA has passed here or ended.
__device__ __forceinline__ void follow_ready() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// close: 0 for an ordinary launch, where other streams' CTAs want the place
// (384 uneven programs, 24 groups of two or three kernels: 3411 us close, 3367 not)
template <class... P, class... A>
cudaError_t launch_following(bool close, void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s,
                             A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute a;
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &a;
  cfg.numAttrs = close ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace sdim
