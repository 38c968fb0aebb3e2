// chain.cuh -- launches of a chain of short kernels on one stream.
//
// On grids of a few 10^4 nodes a kernel of the field solve runs for 3 .. 8 us, and
// an ordinary launch starts it some 2 us after its predecessor has ended.
// launch_chained lets it start while the predecessor's last blocks run: its
// blocks are placed and wait in chain_begin(), which returns once the
// predecessor has completed and its stores are visible.  Every kernel launched
// so calls chain_begin() in all threads before anything else touches memory, so
// the order of the chain is that of ordinary launches; a predecessor that is
// launched in the ordinary way, a copy or an event in between only takes the
// overlap away.
// A step of run_fused in us, with ordinary launches and with these (and the reading
// of the step before moved behind the queued solve): 16^3 at 8 particles per cell
// 238 and 179, 24^3 at 8 325 and 252, 32^3 at 32 296 and 246, 77^3 at 26 1078 and
// 1007.  On large grids the gaps do not count (256 x 128 x 128: 1 % of a step).
//
// What such a kernel reads of its predecessors' results is not declared
// __restrict__: a load through the read-only path is meant for data that does not
// change while the kernel exists, and it exists before they are done.
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

namespace picard {

__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P, class... A>
cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  note_launch();
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace picard
