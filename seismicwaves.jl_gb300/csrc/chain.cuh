// Launches of the time loop as a chain of programmatic dependent launches.
//
// A time step is a chain of two to five short kernels, each reading what the
// one before it wrote.  As plain stream work every link costs the drain of one
// kernel, the launch of the next and its first instructions, one after the
// other (about 1.5 us per link on a GB300 in a CUDA graph, as much as a
// small grid's kernel itself).  Here every kernel of the loop lets its
// successor be scheduled early (chain_next, once all its blocks have called
// it) and waits, as its first action on data that the loop writes, until its
// predecessor has completed and its writes are visible (chain_wait); what lies
// before chain_wait - index arithmetic, shot tables - overlaps with the
// predecessor.  The stencils call chain_next first thing; the source and
// receiver kernels call it after their chain_wait, since their few blocks
// would otherwise let the next stencil in while the previous one still runs,
// and its blocks would crowd on the SMs that became free first (one shot of
// 801 x 801, gradient: 30.4 ms against 36.0; compensated forward of 4 shots of
// 901 x 455: 34.8 against 45.7).  Without any chain_next: 35.3 ms; two shots of
// 601 x 397 elastic, 500 steps: 9.9 ms with, 10.9 without, 16.4 as plain
// launches outside a graph.
//
// Rules that keep the chain safe: a kernel launched with launch_chain calls
// chain_wait in every thread before it returns or touches anything that an
// earlier kernel of the chain reads or writes (so a kernel completes after its
// predecessor, and its successor's wait covers the whole chain); what a kernel
// reads before its wait (shot tables, source time functions, adjoint sources
// and their scale) is written before a full dependency that lies ahead of the
// chain: a copy, a memset or a plainly launched kernel, none of which starts
// before everything ahead of it is complete.  For the adjoint sources, which
// the misfit kernels write, the memsets between these and the adjoint loop are
// that dependency; they may not become chained kernels.  A kernel that reads
// what the loop writes through the read-only path takes its thread index from
// chain_wait_tid.  A kernel launched plainly, a copy or a memset waits for
// everything before it as always, and chain_wait in a plainly launched kernel
// returns at once.
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "internal.h"

namespace swgb {

__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// chain_wait, giving the thread's index in its block.  Loads through the
// read-only path (__ldg, const __restrict__) are invariant to the compiler, so
// no memory clobber keeps it from moving them up past the wait; a load whose
// address is formed with this index cannot move.
__device__ __forceinline__ unsigned chain_wait_tid() {
  unsigned t = threadIdx.x;
  asm volatile("griddepcontrol.wait;" : "+r"(t) : : "memory");
  return t;
}

template <typename... P, typename... Q>
void launch_chain(const char* what, void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t st, Q&&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  check_cuda(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<Q>(args))...), what);
}

}  // namespace swgb
