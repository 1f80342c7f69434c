// pdl.cuh -- programmatic dependent launch.
// A kernel launched with the attribute may be scheduled once every block of
// the kernel ahead of it in the stream has exited; pdl_wait holds it until
// that kernel has completed and its memory is visible.  Without the attribute
// the wait returns at once.  In a chain of such launches every block of every
// kernel waits, so a kernel that has passed its wait sees the results of all
// kernels before it.  No kernel asks for its dependents early
// (griddepcontrol.launch_dependents): a kernel that starts while the ones two
// or three ahead still run may read lines of their vectors that its
// multiprocessor's L1 kept from before (seen as solves that needed a third
// more iterations), and it gained nothing (8^4 FP32 CG 4.2 ms without, 4.4 with).
// Vectors that a kernel ahead writes are plain pointers in these kernels:
// `const ... *__restrict__` would let the compiler read them through the
// read-only path and treat them as unchanging for the kernel's whole life,
// which begins before the wait.  The links, which no kernel of a chain writes,
// keep it, and may be read ahead of the wait.
#pragma once
#include "qopb.h"

namespace qopb {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// pdl: as a dependent of the launch ahead, unless option pdl is 0
template <typename... KArgs, typename... Args>
void launch_k(bool pdl, void (*k)(KArgs...), dim3 grid, dim3 block, cudaStream_t s, Args... args) {
  if (!pdl || !ctx().opt.pdl) {
    k<<<grid, block, 0, s>>>(args...);
    return;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  count_dependents(1);
  QCHECK(cudaLaunchKernelEx(&cfg, k, args...));
}

}  // namespace qopb
