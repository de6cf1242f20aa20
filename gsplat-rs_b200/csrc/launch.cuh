// Kernel launches: what belongs to a device is set once on every device, and a
// launch may have a priority of its own.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <optional>

namespace gsr {

constexpr int kMaxDevices = 64;
inline int current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    cudaGetLastError();
    dev = 0;
  }
  return dev;
}

// Lets kKernel ask for up to `bytes` of dynamic shared memory on the current
// device (the limit is a device's, so a process that renders on several raises
// it on each), with the largest shared memory carve-out if wanted. A call that
// fails is tried again by the next launch; its error stays pending for the
// launch's own check.
template <auto kKernel>
void allow_shared_memory(int bytes, bool max_carveout = false) {
  static std::atomic<bool> done[kMaxDevices];
  const int dev = current_device();
  if (done[dev].load(std::memory_order_relaxed)) return;
  cudaError_t e = cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess && max_carveout)
    e = cudaFuncSetAttribute(kKernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                             cudaSharedmemCarveoutMaxShared);
  if (e == cudaSuccess) done[dev].store(true, std::memory_order_relaxed);
}

// A kernel launch, with a priority of its own where one is given (the priority
// of a captured launch is the launch's, not its stream's). Without one it runs
// at its stream's: a sort on a caller's stream keeps that stream's priority.
template <typename... P, typename... A>
void launch_kernel(void (*kernel)(P...), uint32_t grid, uint32_t threads, size_t smem,
                   std::optional<int> priority, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = stream;
  cudaLaunchAttribute attr{};
  if (priority) {
    attr.id = cudaLaunchAttributePriority;
    attr.val.priority = *priority;
    c.attrs = &attr;
    c.numAttrs = 1;
  }
  cudaLaunchKernelEx(&c, kernel, P(args)...);
}

}  // namespace gsr
