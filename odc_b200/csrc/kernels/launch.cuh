// Launches whose start overlaps the end of the kernel before them on the stream.
//
// A step of a short pack is a chain of kernels of 5-20 us; launch latency and the prologue (barriers, tensor memory, tensor
// maps) of each would otherwise follow the last block of the one before.  A kernel launched with launch_after may become
// resident as soon as every block of its predecessor has called allow_next() or ended, so it calls wait_previous() before
// its first access to global memory: that returns when the predecessor is complete and its writes are visible.  Every such
// kernel waits in every block that does anything, so a predecessor's predecessors are complete as well.  Kernels launched
// without launch_after (other libraries', memsets, the communication kernels) keep the stream's plain order on both sides.
// A kernel that allocates tensor memory calls allow_next() after the allocation: a successor's block must not hold columns
// that a block of its predecessor still waits for.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace odc {

__device__ __forceinline__ void allow_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The same, for pointers that are read through const __restrict__: such a load counts as one of constant memory and could be
// moved above the wait, so the addresses themselves are made to come out of it.
template <typename P0, typename... P>
__device__ __forceinline__ void wait_previous(P0& p0, P&... p) {
  wait_previous();
  asm volatile("" : "+l"(p0) :: "memory");
  ([&] { asm volatile("" : "+l"(p) :: "memory"); }(), ...);
}

template <typename... P, typename... A>
cudaError_t launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  config.attrs = &attr;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, kernel, std::forward<A>(args)...);
}

}  // namespace odc
