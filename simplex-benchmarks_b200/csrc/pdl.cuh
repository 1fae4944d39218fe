// Programmatic dependent launch (sm_90 and later): a kernel may be launched while
// its predecessor on the stream still runs, do what does not depend on it, and
// wait for its completion (and the visibility of its stores) at pdl_wait().
//
// Every kernel launched with launch_pdl calls pdl_wait() before it touches
// anything another kernel writes or reads, and pdl_trigger() only after that.  So
// a kernel's successor starts no earlier than the predecessor's end, and the end
// of a kernel implies the end of everything before it, as in plain stream order.
// A kernel launched without the attribute returns from the wait at once.
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "common.hpp"

namespace sfem {

__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_enter() {
  pdl_wait();
  pdl_trigger();
}

template <class... P, class... A>
inline void launch_pdl(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t lc = {};
  lc.gridDim = dim3(grid);
  lc.blockDim = dim3(block);
  lc.dynamicSmemBytes = smem;
  lc.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  lc.attrs = at;
  lc.numAttrs = 1;
  SFEM_CUDA(cudaLaunchKernelEx(&lc, kernel, P(std::forward<A>(args))...));
}

}  // namespace sfem
