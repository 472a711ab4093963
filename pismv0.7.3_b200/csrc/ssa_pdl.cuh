// ssa_pdl.cuh — programmatic dependent launch between the kernels of a Krylov iteration.
//
// An iteration is a chain of about twenty short kernels, each waiting for the one before.
// A kernel launched with launch_pdl may start while its predecessor still runs: it does what
// does not depend on the predecessor (index arithmetic, loads of the operator), waits in
// pdl_wait() until the predecessor is complete and its writes are visible, and then lets its
// own successor start (pdl_release()).
//
// What may be read before pdl_wait(): because every kernel of the chain releases its successor
// only after its own wait, all kernels but the direct predecessor are complete by then.  So
// anything the direct predecessor does not write.  Everything else, the solver's state with
// its done flag among it, is read after the wait, through a pointer that passed through
// after_wait(), so that no load of it can be moved ahead of the wait.
#pragma once

#include <utility>

#include "ssa_internal.h"

namespace pism_gpu {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// the same pointer, as a value the compiler knows only from here on (!EARLY: in a kernel's form
// that is launched after its predecessor, the pointer as it is)
template <bool EARLY = true, class T>
__device__ __forceinline__ T *after_wait(T *p) {
  if constexpr (EARLY) asm volatile("" : "+l"(p)::"memory");
  return p;
}

// EARLY: while its predecessor still runs; else after it
template <bool EARLY, class... P, class... A>
inline void launch_early(const Launch &L, void (*kernel)(P...), int blocks, int threads, size_t smem, A &&...args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = L.stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = EARLY ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
template <class... P, class... A>
inline void launch_pdl(const Launch &L, void (*kernel)(P...), int blocks, int threads, size_t smem, A &&...args) {
  launch_early<true>(L, kernel, blocks, threads, smem, std::forward<A>(args)...);
}

}  // namespace pism_gpu
