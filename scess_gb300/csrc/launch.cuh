// Kernel launches of the contraction chains.  A residual is some hundred dependent launches,
// many of a few microseconds: each is a programmatic dependent of the one before it, so that
// its blocks are in place, waiting, when that one ends.  An FP64 solve at o = 5, v = 19 (1400
// launches): 11.2 ms with ordinary launches, 9.0 this way; a mixed iteration at o = 10, v = 90 (100):
// 1.82 and 1.67.
#pragma once
#include <cuda_runtime.h>

#include <utility>

#include "common.cuh"

namespace scess {

// First statement of every kernel launched by launch(): lets the next launch be placed once
// all blocks are here, and returns when the launch before is complete and its writes are
// visible.  Every block waits, so a launch never completes before its predecessor.
__device__ __forceinline__ void chain() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... P, typename... A>
void launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A &&...args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  SCESS_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...));
}

}  // namespace scess
