// Kernel launches: every one's result is checked, and what has to be set per device is set on
// each.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <mutex>
#include <utility>

namespace mpsxx {

void cuda_check(cudaError_t e, const char* what);  // engine.cpp

namespace launch_detail {
template <class... P, class... A>
inline void launch(bool chained, void (*k)(P...), dim3 grid, dim3 threads, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = threads;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = chained ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k, P(std::forward<A>(args))...);
  if (e != cudaSuccess) cudaGetLastError();  // reported here, not again by a later call's check
  cuda_check(e, "kernel launch");
}
}  // namespace launch_detail

// Throws where the launch is refused.
template <class... P, class... A>
inline void launch_kernel(void (*k)(P...), dim3 grid, dim3 threads, size_t smem, cudaStream_t st, A&&... args) {
  launch_detail::launch(false, k, grid, threads, smem, st, std::forward<A>(args)...);
}

// Launches k so that its CTAs may be scheduled while the kernel before it on the stream
// drains (programmatic dependent launch).  Such a kernel calls chain_wait() before its first
// access to global memory (it returns once the kernels before have completed and their
// writes are visible), and chain_next() where its successor may be scheduled.
template <class... P, class... A>
inline void launch_chained(void (*k)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A&&... args) {
  launch_detail::launch(true, k, grid, threads, smem, st, std::forward<A>(args)...);
}

constexpr int kLaunchDevices = 64;

// Allows a kernel that much dynamic shared memory on the current device (a limit belongs to
// a device, not to the process).
template <auto K>
inline void allow_smem(size_t bytes) {
  static std::mutex mu;
  static std::atomic<size_t> allowed[kLaunchDevices];
  int dev = 0;
  cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
  const bool known = dev >= 0 && dev < kLaunchDevices;
  if (known && allowed[dev].load(std::memory_order_acquire) >= bytes) return;
  std::lock_guard<std::mutex> lk(mu);
  if (known && allowed[dev].load(std::memory_order_relaxed) >= bytes) return;
  const cudaError_t e = cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
  if (e != cudaSuccess) cudaGetLastError();
  cuda_check(e, "shared memory of a kernel");
  if (known) allowed[dev].store(bytes, std::memory_order_release);
}

#ifdef __CUDACC__
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

}  // namespace mpsxx
