// Launches that overlap the tail of the kernel before them on the stream (programmatic dependent launch).
//
// A kernel launched this way may become resident while its predecessor still runs: as soon as every block of the predecessor has
// called `chain_begin` (or ended) and an SM has room. It runs its set-up and then waits in `chain_begin` until the predecessor has
// completed and its writes are visible, so nothing that an earlier kernel wrote or still reads may be touched before that call, and
// every thread of every chained kernel makes it (a block that left without it could let the kernel after next start too early).
// What it saves is the gap between two dependent launches: about 4 us between GEMMs of one stream (2 us of it the set-up of a CTA
// pair), in chains of kernels of 5 to 50 us.
//
// Kernels that may wait for another GPU are launched plainly and call `chain_wait` instead, so that their successor starts when they have
// ended. Let in early it would hold every SM that they leave free (a GEMM: all of its shared memory) for as long as the peer is late, and
// work of other streams, which the peer may be waiting for in turn, would have none.
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace tb {

__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_begin() {
  chain_wait();
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... Params, typename... Args>
inline cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace tb
