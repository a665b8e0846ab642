// Kernel launches of a dependent chain (programmatic dependent launch).
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace mpsxx {

// Launches k so that its CTAs may be scheduled while the kernel before it on the stream
// drains.  Such a kernel calls chain_wait() before its first access to global memory (it
// returns once the kernels before have completed and their writes are visible), and
// chain_next() where its successor may be scheduled.
template <class... P, class... A>
inline void launch_chained(void (*k)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A&&... args) {
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
  cudaLaunchKernelEx(&cfg, k, P(std::forward<A>(args))...);
}

#ifdef __CUDACC__
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

}  // namespace mpsxx
