// Launches of kernels that follow one another on a stream (the passes of a transform, the steps of a prover call).
//
// Each such kernel is launched with programmatic stream serialization: it may start while the kernel before it on the
// stream drains, and waits at chain_wait() until that one has ended and its writes are visible.  Every thread of a
// kernel launched this way calls chain_wait() before it touches global memory that any kernel writes, also a thread
// without work: a kernel's end then implies the end of all before it.  What an earlier kernel wrote is read with
// ld.global.cg, and no pointer to it is const __restrict__: such loads might be moved ahead of the wait.
// chain_next() lets the following kernel be set up once every block of this one has called it or ended (a kernel without
// it, a caller's own, is followed only at its end).  It stands before a block's last stores, not at its start: blocks
// set up early wait on whatever SMs have room, and a small pass then left its successor unevenly placed (BLS12-381 QAP
// of 2^16, 22 launches: 202 us without the chain, 312 with the call at the start).
#pragma once
#include <cuda_runtime.h>

namespace gsn {

__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... Params, class... Args>
inline cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid, unsigned block, size_t smem, cudaStream_t s,
                                  Args... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

}  // namespace gsn
