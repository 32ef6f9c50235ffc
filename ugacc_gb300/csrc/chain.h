// Launches that overlap with the end of the kernel before them in the stream.
//
// A solve at no=5/nv=19 is some hundred kernels of 2 to 10 us in a row, with 2.2 to 2.7 us between
// one's end and the next one's first instruction.  A kernel launched with launch_chained starts
// when its predecessor's blocks have ended, without waiting for the flush of their writes; that
// wait is in chain_enter(), in each block.  Solves (median, plain launches -> chained):
// CCSD no=5/nv=19 2.22 -> 1.65 ms, its Lambda and densities 3.43 -> 2.59 ms, a gradient at
// no=5/nv=24 10.2 -> 8.2 ms, six perturbed solves and the response functions at no=6/nv=22
// 23.6 -> 17.7 ms.  No kernel lets its successor start earlier (launch_dependents): the waiting
// blocks of several successors then held places on the SMs, those that started next were spread
// unevenly, and the same four took 1.82, 3.10, 10.6 and 19.7 ms, or, with the signal after a
// GEMM's main loop only, 1.69, 2.74, 8.7 and 18.4 ms.
//
// Rules: chain_enter() is the first statement, before any access to global memory.  As every
// kernel of a chain waits for its predecessor's end, the wait covers all that came before.  The
// kernel's pointers are not __restrict__, nor are those of the functions inlined into it: what is
// read through such a pointer could be fetched ahead of the wait.  A launch without the attribute, a copy or an event between two kernels
// waits as always.
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "core.h"

namespace ucc {

__device__ __forceinline__ void chain_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// cluster: CTAs of a cluster along x (1: none)
template <typename... P, typename... A>
void launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t stream, unsigned cluster, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  UCC_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}

}  // namespace ucc
