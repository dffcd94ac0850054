// Kernel launches in the stream's plain order.
//
// Overlapped starts (programmatic stream serialisation: a kernel becomes resident while the one before it still runs) took
// 4 % off the smallest training step (2295 -> 2190 us).  They are not used: long chains of token log-probabilities, forward
// and backward, twice stopped making progress on the GPU with them, and never without.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace odc {

template <typename... P, typename... A>
cudaError_t launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchConfig_t config{};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  return cudaLaunchKernelEx(&config, kernel, std::forward<A>(args)...);
}

}  // namespace odc
