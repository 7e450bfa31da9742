// Programmatic dependent launch: a kernel of a chain is scheduled while its predecessor drains, so
// its launch latency and what it reads of data that no kernel of the chain writes (index maps) lie
// under the predecessor's last wave.  Every kernel launched with launch_dependent() calls
// pdl_trigger() first (its own successor may be scheduled) and pdl_wait() before it touches memory
// that the chain writes: the wait returns when the predecessor has completed and its writes are
// visible, and a predecessor completes only after its own wait, so the order of the whole chain
// is that of the stream.
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "pmg_internal.hpp"

namespace pmg {

__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// p as a value that exists only after the wait, for loads the compiler may otherwise move before it
// (inline PTX, const __restrict__ pointers).  What the chain writes is read with plain loads, not
// through the non-coherent path: it changes while the waiting kernel is resident.
template <typename T> __device__ __forceinline__ T *pdl_after(T *p) {
  asm volatile("" : "+l"(p));
  return p;
}

template <typename... P, typename... A>
void launch_dependent(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, A &&...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  PMG_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}

} // namespace pmg
