// ssa_control.cu — device-side control of the Picard loop.
//
// A whole SSAFD solve (SSAFD::picard_manager, SSAFD.cc:962-1119, with its linear solves) can
// run as one CUDA graph whose conditional WHILE / IF nodes take their values from a PState
// in device memory.  These single-thread kernels make the decisions the host loop makes, in
// the same double arithmetic, so the graph takes the same path: the KSP tolerance of each
// Picard iteration (inexact Picard), the refinement steps of the mixed-precision solve, the
// zero-diagonal and KSP-failure checks and the Picard stopping test (SSAFD.cc:1084).  The
// decisions themselves are the __host__ __device__ functions of ssa_state.h; these kernels
// apply them to the state in device memory.
#include <climits>

#include "ssa_pdl.cuh"

namespace pism_gpu {
namespace {

// picard_loop: the WHILE node over Picard passes, entered
__global__ void k_picard_start(PState *P, cudaGraphConditionalHandle picard_loop) {
  picard_start(*P);
  cudaGraphSetConditional(picard_loop, 1u);
}

// mixed precision: refine_loop (the WHILE node over refinement steps) is entered; FP64: st is
// made ready for the solve
__global__ void k_picard_begin(PState *P, PicardConst c, int *zero_diag_cell, cudaGraphConditionalHandle refine_loop,
                               KState *st, int maxit) {
  *zero_diag_cell = INT_MAX;
  picard_begin(*P, c);
  if (st) ksp_begin(*st, *P, maxit);
  else cudaGraphSetConditional(refine_loop, 1u);
}

__global__ void k_refine_end(PState *P, const KState *st, int max_refine) {
  pdl_release();
  refine_end(*P, *st, max_refine);
}

// st: the FP64 solve's state (body_iters iterations a pass of its loop), else null
__global__ void k_picard_after_solve(PState *P, const int *zero_diag_cell, const KState *st, int body_iters) {
  pdl_release();
  if (st) ksp_end(*P, *st, body_iters);
  picard_after_solve(*P, *zero_diag_cell);
}

// after the nu*H update (neither does anything once the solve failed); picard_loop goes on or ends
__global__ void k_picard_test(PState *P_, const double *norm2_, PicardConst c, cudaGraphConditionalHandle picard_loop) {
  pdl_wait();
  PState *P = after_wait(P_);
  const double *norm2 = after_wait(norm2_);
  if (!P->done) picard_test(*P, norm2[0], norm2[1], c);
  cudaGraphSetConditional(picard_loop, P->done ? 0u : 1u);
}

__global__ void k_flag_condition(cudaGraphConditionalHandle cond, const int *flag) {
  cudaGraphSetConditional(cond, *flag != 0 ? 1u : 0u);
}

}  // namespace

void launch_picard_start(const Launch &L, PState *P, cudaGraphConditionalHandle picard_loop) {
  L.tick();
  k_picard_start<<<1, 1, 0, L.stream>>>(P, picard_loop);
}
void launch_picard_begin(const Launch &L, PState *P, const PicardConst &c, int *zero_diag_cell,
                         cudaGraphConditionalHandle refine_loop, KState *st, int maxit) {
  L.tick();
  k_picard_begin<<<1, 1, 0, L.stream>>>(P, c, zero_diag_cell, refine_loop, st, maxit);
}
void launch_refine_end(const Launch &L, PState *P, const KState *st, int max_refine) {
  L.tick();
  k_refine_end<<<1, 1, 0, L.stream>>>(P, st, max_refine);
}
void launch_picard_after_solve(const Launch &L, PState *P, const int *zero_diag_cell, const KState *st,
                               int body_iters) {
  L.tick();
  k_picard_after_solve<<<1, 1, 0, L.stream>>>(P, zero_diag_cell, st, body_iters);
}
void launch_picard_test(const Launch &L, PState *P, const double *norm2, const PicardConst &c,
                        cudaGraphConditionalHandle picard_loop) {
  L.tick();
  launch_pdl(L, k_picard_test, 1, 1, 0, P, norm2, c, picard_loop);
}
void launch_flag_condition(const Launch &L, cudaGraphConditionalHandle cond, const int *flag) {
  L.tick();
  k_flag_condition<<<1, 1, 0, L.stream>>>(cond, flag);
}

}  // namespace pism_gpu
