// Launches of kernels that follow one another in a stream.
//
// A query is a chain of short kernels (a step of the filter or of the joins
// takes 5-50 us), and each waits 1-2 us between the last block of the one
// before and its own first. Launched this way (programmatic dependent launch),
// a kernel's blocks are set up while the kernel before drains, and wait at
// wait_for_previous() until it has completed and its writes are visible.
// B200: the filter of queries on the 2^22-vertex R-MAT graph 3.95 -> 3.62 ms,
// a batch of 12-vertex queries on 2^20 vertices 25.5 -> 23.6 ms, one such
// query 2.70 -> 2.54 ms; batches that run a dozen queries at once have no such
// gaps and take what they took.
//
// Every kernel launched by launch_next calls wait_for_previous() first, before
// it touches memory, in every thread: so a kernel that completes has seen the
// one before it complete, and the order of the stream holds through the chain.
// (Signalling the next kernel earlier, at a kernel's start, filled SMs with
// waiting blocks and gained nothing more.)
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "internal.h"

namespace gpsm {

#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
void launch_next(void (*kernel)(P...), dim3 grid, uint32_t block, cudaStream_t s, A&&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3(block);
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  GPSM_CUDA(cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...));
}
#endif

}  // namespace gpsm
