// Launches that overlap the end of the kernel before them on their stream (programmatic dependent launch), for the chain of
// short kernels of a decoding step: a kernel launched this way may start while its predecessor still runs, so it
//   * calls wait_predecessors() before it touches global memory (after it, every earlier kernel of the stream is complete and
//     its writes are visible);
//   * calls allow_dependents() when its own loads are on their way: a successor launched the same way then gets its blocks as soon
//     as all of this kernel's blocks have come so far.
// Measured on a decoding step of 6 layers of 2048 in a replayed graph: 301 -> 285 us. Fetching a product's weight into L2
// ahead of the wait, by bulk or by line, made the step slower (332 to 345 us), and so did allow_dependents() at the start of the
// products (292 us): what comes early takes bandwidth and blocks from the kernel that everything waits for.
// A kernel launched the ordinary way waits for its predecessors as ever. Captured launches keep the relation in the graph.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace tb {

__device__ __forceinline__ void wait_predecessors() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename... P, typename... A>
cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t stream, A&&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);
}

}  // namespace tb
