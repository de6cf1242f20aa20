// A kernel launch with a priority of its own. The priority of a captured launch
// is the launch's, not its stream's.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace gsr {

template <typename... P, typename... A>
void launch_kernel(void (*kernel)(P...), uint32_t grid, uint32_t threads, size_t smem,
                   int priority, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributePriority;
  attr.val.priority = priority;
  c.attrs = &attr;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, P(args)...);
}

}  // namespace gsr
