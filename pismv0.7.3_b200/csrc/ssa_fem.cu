// ssa_fem.cu — the Q1 finite-element SSA (SSAFEM.cc:151-840, FETools.cc/.hh) on the GPU:
// the coefficients cached at the 2 x 2 Gauss points of each element
// (SSAFEM::cacheQuadPtValues, SSAFEM.cc:233-375), the weak-form residual
// (compute_local_function, :441-532) and its Newton Jacobian (compute_local_jacobian,
// :571-700), Dirichlet rows scale (u - u_bc) with their columns dropped (DirichletData_Vector,
// FETools.cc:671-741), and the linear solves of the Newton steps by conjugate gradients with
// the inverse 2 x 2 diagonal blocks as preconditioner.
//
// Layout: the residual and Jacobian are assembled per node, not per element.  One thread owns
// node (i, j) and walks the (up to) four elements around it in the reference's element order
// ((i-1, j-1), (i-1, j), (i, j-1), (i, j): i outer), computing each element's quadrature
// values and adding the element's row block for this node, so the sums are deterministic and
// no element buffer or atomic is needed; the price is each element's quadrature evaluated by
// its four nodes.  The Jacobian is stored as 9 neighbour blocks of 2 x 2 per node,
// structure-of-arrays ([36][N]), which the CG apply reads coalesced.
#include <algorithm>
#include <climits>

#include "ssa_exchange.cuh"
#include "ssa_fem.h"
#include "ssa_reduce.cuh"

namespace pism_gpu {

namespace {

constexpr int NTF = RED_THREADS;

// the element-local node offsets of DOFMap (FETools.cc:206-207)
__constant__ int kDI[4] = {0, 1, 1, 0};
__constant__ int kDJ[4] = {0, 0, 1, 1};

struct FemGrid {
  int Mx, My, nex, ney, px, py;   // px, py: periodic in x / y
};

__device__ __forceinline__ int fem_node(const FemGrid &G, int i, int j) {
  return wrap(i, G.Mx) * G.My + wrap(j, G.My);
}

// FlowLaw::averaged_hardness (flowlaws.cc:141-185) over the enthalpy column interpolated to a
// quadrature point from the element's four node columns, Enth_q[k] = sum_p val[p] E_p[k]
// (SSAFEM.cc:326-339)
__device__ double fem_averaged_hardness(const pism_gpu_ssa_config &c, double H, const double *z, int Mz,
                                        const double *E[4], const double val[4]) {
  int kb = 0, hi = Mz - 1;   // kBelowHeight: largest k in [0, Mz-2] with z[k] <= H
  while (hi > kb + 1) {
    const int mid = (kb + hi) / 2;
    if (z[mid] > H) hi = mid; else kb = mid;
  }
  auto Eq = [&](int k) {
    double e = 0.0;
    for (int p = 0; p < 4; ++p) e += val[p] * E[p][k];
    return e;
  };
  double B = 0.0;
  if (kb > 0) {
    double h0 = hardness_parameter(c, Eq(0), ec_pressure(c, H));
    for (int k = 1; k <= kb; ++k) {
      const double h1 = hardness_parameter(c, Eq(k), ec_pressure(c, H - z[k]));
      B += (z[k] - z[k - 1]) * (h0 + h1);
      h0 = h1;
    }
  }
  B *= 0.5;
  const double depth = H - z[kb];
  B += depth * hardness_parameter(c, Eq(kb), ec_pressure(c, depth));
  return H > 0 ? B / H : 0.0;
}

// SSAFEM::cacheQuadPtValues (SSAFEM.cc:233-375): one thread per element
__global__ void __launch_bounds__(NTF) k_fem_coefficients(FemGrid G, pism_gpu_ssa_config c, FemGerms W,
                                                          FemCoef C, const double *H, const double *bed,
                                                          const double *tauc, const double *srf,
                                                          const double *enthalpy, const double *z, int Mz,
                                                          double icefree_thickness, double is_floating_thickness) {
  const int Ne = G.nex * G.ney;
  const double alpha = 1.0 - c.ice_density / c.sea_water_density;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < Ne; e += gridDim.x * blockDim.x) {
    const int ei = e / G.ney, ej = e - ei * G.ney;
    int n[4];
    for (int k = 0; k < 4; ++k) n[k] = fem_node(G, ei + kDI[k], ej + kDJ[k]);
    for (int q = 0; q < 4; ++q) {
      double Hq = 0, bq = 0, tq = 0, hx = 0, hy = 0;
      for (int k = 0; k < 4; ++k) {   // Quadrature_Scalar::computeTrialFunctionValues
        Hq += W.val[q][k] * H[n[k]];
        bq += W.val[q][k] * bed[n[k]];
        tq += W.val[q][k] * tauc[n[k]];
        hx += W.gx[q][k] * srf[n[k]];
        hy += W.gy[q][k] * srf[n[k]];
      }
      const int o = q * Ne + e;
      C.H[o] = Hq;
      C.tauc[o] = tq;
      C.tdu[o] = -c.ice_density * c.standard_gravity * Hq * hx;
      C.tdv[o] = -c.ice_density * c.standard_gravity * Hq * hy;
      // GeometryCalculator::mask (Mask.hh:82-118), dry simulation off
      const double hgrounded = bq + Hq, hfloating = c.sea_level + alpha * Hq;
      const bool floating = hfloating > hgrounded + is_floating_thickness, ice_free = Hq < icefree_thickness;
      C.mask[o] = (int8_t)(floating ? (ice_free ? MASK_ICE_FREE_OCEAN : MASK_FLOATING)
                                    : (ice_free ? MASK_ICE_FREE_BEDROCK : MASK_GROUNDED));
      if (c.flow_law == PISM_FLOW_LAW_ISOTHERMAL_GLEN) {
        C.B[o] = pow(c.ice_softness, -1.0 / c.ssa_Glen_exponent);
      } else {
        const double *E[4] = {enthalpy + (size_t)n[0] * Mz, enthalpy + (size_t)n[1] * Mz,
                              enthalpy + (size_t)n[2] * Mz, enthalpy + (size_t)n[3] * Mz};
        C.B[o] = fem_averaged_hardness(c, Hq, z, Mz, E, W.val[q]);
      }
    }
  }
}

// SSAFEM::PointwiseNuHAndBeta (SSAFEM.cc:393-432) with FlowLaw::effective_viscosity
// (flowlaws.hh:100-112) and drag_with_derivative (basal_resistance.cc:59-68, 174-190)
struct Pointwise {
  double eta, deta, beta, dbeta;
};

__device__ __forceinline__ Pointwise nuH_and_beta(const FemProblem &P, double H, double B, double tauc, int mask,
                                                  double u, double v, const double Du[3]) {
  const pism_gpu_ssa_config &c = P.c;
  Pointwise w;
  if (H < c.min_thickness_strength_extension_ssa) {
    w.eta = P.notional_strength;
    w.deta = 0.0;
  } else {
    const double n = c.ssa_Glen_exponent, power = (1.0 - n) / (2.0 * n);
    const double reg = (c.Schoof_regularizing_velocity / c.Schoof_regularizing_length) *
                       (c.Schoof_regularizing_velocity / c.Schoof_regularizing_length);
    // secondInvariantDu_2D, flowlaws.hh:42-44
    const double gamma = 0.5 * (Du[0] * Du[0] + Du[1] * Du[1] + (Du[0] + Du[1]) * (Du[0] + Du[1]) +
                                2 * Du[2] * Du[2]);
    const double nu = 0.5 * B * pow(reg + gamma, power);
    w.eta = c.epsilon_ssa + nu * H;
    w.deta = power * nu / (reg + gamma) * H;
  }
  if (m_grounded_ice(mask)) {
    const double magreg2 = c.plastic_regularization * c.plastic_regularization + u * u + v * v;
    if (!c.do_pseudo_plastic_till) {
      w.beta = tauc / sqrt(magreg2);
      w.dbeta = -1 * w.beta / magreg2;
    } else {
      const double q = c.pseudo_plastic_q;
      if (c.sliding_scale_factor_reduces_tauc > 0.0) {
        const double Aq = pow(c.sliding_scale_factor_reduces_tauc, q);
        w.beta = (tauc / Aq) * pow(magreg2, 0.5 * (q - 1)) * pow(c.pseudo_plastic_uthreshold, -q);
      } else {
        w.beta = tauc * pow(magreg2, 0.5 * (q - 1)) * pow(c.pseudo_plastic_uthreshold, -q);
      }
      w.dbeta = (q - 1) * w.beta / magreg2;
    }
  } else {
    w.beta = m_ice_free_land(mask) ? c.beta_ice_free_bedrock : 0.0;
    w.dbeta = 0.0;
  }
  return w;
}

// The residual (compute_local_function, SSAFEM.cc:441-532) and, with JAC, the Jacobian rows
// (compute_local_jacobian, :571-700) of one node, summed over its elements in the reference's
// element order; ||F||^2 over the grid in block order.
template <bool JAC>
__global__ void __launch_bounds__(NTF) k_fem_node(FemProblem P, FemGrid G, FemCoef C, const double2 *vel,
                                                  const uint8_t *bc, const double2 *bcv, double2 *F, double *J,
                                                  double4 *dinv, int *zero_pivot, FemScalars *sc,
                                                  double *partials, unsigned *ticket) {
  const int N = G.Mx * G.My, Ne = G.nex * G.ney;
  const FemGerms &W = P.W;
  double acc[1] = {0.0};
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
    const int i = n / G.My, j = n - i * G.My;
    double Jn[9][2][2];
    if (JAC)
      for (int b = 0; b < 9; ++b) Jn[b][0][0] = Jn[b][0][1] = Jn[b][1][0] = Jn[b][1][1] = 0.0;
    double2 Fn = make_double2(0.0, 0.0);
    if (bc[n]) {   // DirichletData_Vector::fix_residual / fix_jacobian (FETools.cc:702-741)
      const double2 x = vel[n], b = bcv[n];
      Fn = make_double2(P.scale * (x.x - b.x), P.scale * (x.y - b.y));
      if (JAC) Jn[4][0][0] = Jn[4][1][1] = P.scale;
    } else {
      // the elements around the node, in element order; k: the node's place in each
      const int erel[4][2] = {{-1, -1}, {-1, 0}, {0, -1}, {0, 0}};
      const int kloc[4] = {2, 1, 3, 0};
      for (int t = 0; t < 4; ++t) {
        int ei = i + erel[t][0], ej = j + erel[t][1];
        if (G.px) ei = wrap(ei, G.Mx); else if (ei < 0 || ei >= G.nex) continue;
        if (G.py) ej = wrap(ej, G.My); else if (ej < 0 || ej >= G.ney) continue;
        const int e = ei * G.ney + ej, k = kloc[t];
        double2 xl[4];
        bool lbc[4];
        for (int l = 0; l < 4; ++l) {   // DirichletData_Vector::update (FETools.cc:680-692)
          const int nl = fem_node(G, ei + kDI[l], ej + kDJ[l]);
          lbc[l] = bc[nl] != 0;
          xl[l] = lbc[l] ? bcv[nl] : vel[nl];
        }
        double ru = 0.0, rv = 0.0;
        double K[2][4][2];
        if (JAC)
          for (int l = 0; l < 4; ++l) K[0][l][0] = K[0][l][1] = K[1][l][0] = K[1][l][1] = 0.0;
        for (int q = 0; q < 4; ++q) {
          // Quadrature_Vector::computeTrialFunctionValues (FETools.cc:431-446)
          double u = 0, v = 0, Du[3] = {0, 0, 0};
          for (int l = 0; l < 4; ++l) {
            u += W.val[q][l] * xl[l].x;
            v += W.val[q][l] * xl[l].y;
            Du[0] += W.gx[q][l] * xl[l].x;
            Du[1] += W.gy[q][l] * xl[l].y;
            Du[2] += 0.5 * (W.gy[q][l] * xl[l].x + W.gx[q][l] * xl[l].y);
          }
          const int o = q * Ne + e;
          const Pointwise pw = nuH_and_beta(P, C.H[o], C.B[o], C.tauc[o], C.mask[o], u, v, Du);
          const double jw = W.JxW[q];
          const double Ux = Du[0], Vy = Du[1], UyVx = 2.0 * Du[2];
          const double psi = W.val[q][k], psx = W.gx[q][k], psy = W.gy[q][k];
          const double tbu = u * (-pw.beta), tbv = v * (-pw.beta);
          ru += jw * (pw.eta * (psx * (4.0 * Ux + 2.0 * Vy) + psy * UyVx) - psi * (tbu + C.tdu[o]));
          rv += jw * (pw.eta * (psx * UyVx + psy * (2.0 * Ux + 4.0 * Vy)) - psi * (tbv + C.tdv[o]));
          if (JAC) {
            for (int l = 0; l < 4; ++l) {
              const double phi = W.val[q][l], phx = W.gx[q][l], phy = W.gy[q][l];
              const double gamma_u = (2.0 * Ux + Vy) * phx + Du[2] * phy;
              const double gamma_v = Du[2] * phx + (Ux + 2.0 * Vy) * phy;
              const double eta_u = pw.deta * gamma_u, eta_v = pw.deta * gamma_v;
              const double taub_xu = -pw.dbeta * u * u * phi - pw.beta * phi;
              const double taub_xv = -pw.dbeta * u * v * phi;
              const double taub_yu = -pw.dbeta * v * u * phi;
              const double taub_yv = -pw.dbeta * v * v * phi - pw.beta * phi;
              K[0][l][0] += jw * (eta_u * (psx * (4 * Ux + 2 * Vy) + psy * UyVx) +
                                  pw.eta * (4 * psx * phx + psy * phy) - psi * taub_xu);
              K[0][l][1] += jw * (eta_v * (psx * (4 * Ux + 2 * Vy) + psy * UyVx) +
                                  pw.eta * (2 * psx * phy + psy * phx) - psi * taub_xv);
              K[1][l][0] += jw * (eta_u * (psx * UyVx + psy * (2 * Ux + 4 * Vy)) +
                                  pw.eta * (psx * phy + 2 * psy * phx) - psi * taub_yu);
              K[1][l][1] += jw * (eta_v * (psx * UyVx + psy * (2 * Ux + 4 * Vy)) +
                                  pw.eta * (psx * phx + 4 * psy * phy) - psi * taub_yv);
            }
          }
        }
        Fn.x += ru;   // DOFMap::addLocalResidualBlock
        Fn.y += rv;
        if (JAC)
          for (int l = 0; l < 4; ++l) {
            if (lbc[l]) continue;   // Dirichlet columns are left out (DirichletData::constrain)
            const int b = (erel[t][0] + kDI[l] + 1) * 3 + (erel[t][1] + kDJ[l] + 1);
            Jn[b][0][0] += K[0][l][0];
            Jn[b][0][1] += K[0][l][1];
            Jn[b][1][0] += K[1][l][0];
            Jn[b][1][1] += K[1][l][1];
          }
      }
    }
    F[n] = Fn;
    acc[0] += Fn.x * Fn.x + Fn.y * Fn.y;
    if (JAC) {
      for (int b = 0; b < 9; ++b)
        for (int r = 0; r < 2; ++r)
          for (int s = 0; s < 2; ++s) J[(size_t)(b * 4 + r * 2 + s) * N + n] = Jn[b][r][s];
      const double a = Jn[4][0][0], b = Jn[4][0][1], cc = Jn[4][1][0], d = Jn[4][1][1];
      const double det = a * d - b * cc;
      if (det == 0.0 || !isfinite(det)) {
        *zero_pivot = n + 1;
        dinv[n] = make_double4(0.0, 0.0, 0.0, 0.0);
      } else {
        dinv[n] = make_double4(d / det, -b / det, -cc / det, a / det);
      }
    }
  }
  double tot[1];
  if (grid_reduce<1>(acc, partials, ticket, tot)) sc->f2 = tot[0];
}

// ---- conjugate gradients on J du = -F, preconditioned by the inverse diagonal blocks ----
// Which product of a sum is rounded by itself is written out, so that the kernels of an iteration
// and the one of a whole solve give the same bits (left to the compiler they did not: 289 and 287
// iterations of the first linear solve on 5 x 481 nodes): a b + c d with c d rounded first.
__device__ __forceinline__ double two(double a, double b, double c, double d) {
  return __fma_rn(a, b, __dmul_rn(c, d));
}
__device__ __forceinline__ double dot(const double2 &a, const double2 &b) { return two(a.x, b.x, a.y, b.y); }
__device__ __forceinline__ double2 axpy(double s, const double2 &x, const double2 &y) {
  return make_double2(__fma_rn(s, x.x, y.x), __fma_rn(s, x.y, y.y));
}
__device__ __forceinline__ double2 bmul(const double4 &A, const double2 &x) {
  return make_double2(two(A.x, x.x, A.y, x.y), two(A.z, x.x, A.w, x.y));
}

__global__ void __launch_bounds__(NTF) k_cg_init(int N, const double2 *F, const double4 *dinv, double2 *x,
                                                 double2 *r, double2 *z, double2 *p, FemCG *cg, double rtol,
                                                 int maxit, double *partials, unsigned *ticket) {
  double acc[2] = {0.0, 0.0};
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
    const double2 rn = make_double2(-F[n].x, -F[n].y);
    const double4 A = dinv[n];   // (here the other product first, as this kernel has always rounded)
    const double2 zn = make_double2(two(A.y, rn.y, A.x, rn.x), two(A.w, rn.y, A.z, rn.x));
    x[n] = make_double2(0.0, 0.0);
    r[n] = rn;
    z[n] = zn;
    p[n] = zn;
    acc[0] += two(rn.y, zn.y, rn.x, zn.x);
    acc[1] += two(rn.y, rn.y, rn.x, rn.x);
  }
  double tot[2];
  if (grid_reduce<2>(acc, partials, ticket, tot)) {
    cg->rz = tot[0];
    cg->bb = tot[1];
    cg->rr = tot[1];
    cg->rtol = rtol;
    cg->maxit = maxit;
    cg->its = 0;
    cg->done = tot[1] == 0.0 ? 1 : 0;
  }
}

__global__ void __launch_bounds__(NTF) k_cg_apply(FemGrid G, const double *J, const double2 *p, double2 *q,
                                                  FemCG *cg, double *partials, unsigned *ticket) {
  if (cg->done) return;   // uniform over the grid: set by an earlier kernel
  const int N = G.Mx * G.My;
  double acc[1] = {0.0};
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
    const int i = n / G.My, j = n - i * G.My;
    double2 y = make_double2(0.0, 0.0);
    for (int b = 0; b < 9; ++b) {
      const double2 x = p[fem_node(G, i + b / 3 - 1, j + b % 3 - 1)];
      y.x += two(J[(size_t)(b * 4 + 0) * N + n], x.x, J[(size_t)(b * 4 + 1) * N + n], x.y);
      y.y += two(J[(size_t)(b * 4 + 2) * N + n], x.x, J[(size_t)(b * 4 + 3) * N + n], x.y);
    }
    q[n] = y;
    const double2 pn = p[n];
    acc[0] += dot(pn, y);
  }
  double tot[1];
  if (grid_reduce<1>(acc, partials, ticket, tot)) {
    cg->pq = tot[0];
    if (!(tot[0] > 0.0)) cg->done = 2;   // J not positive definite along p
    else cg->alpha = cg->rz / tot[0];
  }
}

__global__ void __launch_bounds__(NTF) k_cg_update(int N, const double4 *dinv, const double2 *p, const double2 *q,
                                                   double2 *x, double2 *r, double2 *z, FemCG *cg, double *partials,
                                                   unsigned *ticket) {
  if (cg->done) return;
  const double alpha = cg->alpha;
  double acc[2] = {0.0, 0.0};
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
    const double2 pn = p[n], qn = q[n];
    const double2 rn = axpy(-alpha, qn, r[n]), zn = bmul(dinv[n], rn);
    x[n] = axpy(alpha, pn, x[n]);
    r[n] = rn;
    z[n] = zn;
    acc[0] += dot(rn, zn);
    acc[1] += dot(rn, rn);
  }
  double tot[2];
  if (grid_reduce<2>(acc, partials, ticket, tot)) {
    cg->beta = tot[0] / cg->rz;
    cg->rz = tot[0];
    cg->rr = tot[1];
    cg->its += 1;
    if (tot[1] <= cg->rtol * cg->rtol * cg->bb) cg->done = 1;
    else if (cg->its >= cg->maxit) cg->done = 3;
  }
}

__global__ void __launch_bounds__(NTF) k_cg_direction(int N, const double2 *z, double2 *p, const FemCG *cg) {
  if (cg->done) return;
  const double beta = cg->beta;
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
    p[n] = axpy(beta, p[n], z[n]);
  }
}

// The whole CG solve in one cooperative kernel, one thread a node: the node's 36 Jacobian
// coefficients and the p its block reads in shared memory, its x, r and z in registers.  An
// iteration costs two exchanges (ssa_exchange.cuh): (p, q), then (r, z) and (r, r); then the z
// around the block are read from words of their own, and the block updates its copies of the
// neighbours' p as their owners do.
//
// A block owns NTF nodes in a row of the linear order, from s0 on.  The p its stencils read lie in
// three runs of NTF + 2 nodes, from s0 - My - 1, s0 - 1 and s0 + My - 1 (modulo N: the grid's rows
// wrap), but for a neighbour of a node at a row's end, or two of the last node's, which that
// thread keeps by itself.
//
// Bound: the two exchanges' and the halo's trips through L2; the Jacobian's 288 B a node come from
// shared memory.  One B200, three kernels an iteration / this kernel: 5 x 481 nodes 12.5 / 4.5 us
// an iteration, 241 x 241 15.3 / 7.4 us.  The same operations per node and the same order of the
// sums as those kernels, which remain for the grids that do not fit (more than two blocks an SM,
// 75 776 nodes on 148).
constexpr int CG_RUN = NTF + 2;
constexpr int CG_SMEM = 36 * NTF * (int)sizeof(double) + 3 * CG_RUN * (int)sizeof(double2);

template <class Limit>
__global__ void __launch_bounds__(NTF, 2) k_cg_resident(FemGrid G, const double *__restrict__ J,
                                                        const double4 *__restrict__ dinv,
                                                        const double2 *__restrict__ r0, const double2 *__restrict__ z0,
                                                        double2 *__restrict__ x_out, ExNodes<Limit> zex, FemCG *cg,
                                                        ExSlots<Limit> slots_q, ExSlots<Limit> slots_r) {
  extern __shared__ __align__(16) double Js[];   // [36][NTF], then the three runs of p
  double2 *const P = reinterpret_cast<double2 *>(Js + 36 * NTF);
  const int N = G.Mx * G.My, tid = threadIdx.x, s0 = blockIdx.x * NTF, n = s0 + tid;
  const bool mine = n < N;
  const int i = mine ? n / G.My : 0, j = mine ? n - i * G.My : 0;
  auto modN = [&](int k) { return (k % N + N) % N; };
  const int base[3] = {s0 - G.My - 1, s0 - 1, s0 + G.My - 1};
  // each neighbour's place in the runs; -1, -2: the node apart[0], apart[1], kept by this thread
  short at[9];
  int apart[2] = {-1, -1};
  bool lone = false;
#pragma unroll
  for (int b = 0; b < 9; ++b) {
    const int m = mine ? fem_node(G, i + b / 3 - 1, j + b % 3 - 1) : 0;
    int place = -1;
#pragma unroll
    for (int q = 2; q >= 0; --q) {
      const int k = modN(m - base[q]);
      // the middle run is the block's own nodes and one on either side
      if (k < CG_RUN && (q != 1 || k == 0 || k == CG_RUN - 1 || s0 + k - 1 < N)) place = q * CG_RUN + k;
    }
    if (mine && place < 0) {
      if (apart[0] < 0 || apart[0] == m) {
        apart[0] = m;
      } else {
        lone = lone || (apart[1] >= 0 && apart[1] != m);
        apart[1] = m;
        place = -2;
      }
    }
    at[b] = (short)place;
  }
  // what this thread reads into the runs: above and below its node; six threads a run's end each
  const int above = modN(base[0] + tid), below = modN(base[2] + tid), e = tid - (NTF - 6);
  const int end_run = e >> 1, end_k = e < 0 ? -1 : (end_run == 1 ? (e & 1) * (NTF + 1) : NTF + (e & 1));
  const int end = e < 0 ? -1 : modN(base[end_run] + end_k), end_at = end_run * CG_RUN + end_k;
  const bool more = __any_sync(0xffffffffu, apart[0] >= 0 || end >= 0);
  double2 x = make_double2(0.0, 0.0), r = x, z = x;   // p starts as z
  double2 pa = apart[0] >= 0 ? z0[apart[0]] : x, pa2 = apart[1] >= 0 ? z0[apart[1]] : x;
  double4 d = make_double4(0.0, 0.0, 0.0, 0.0);
  P[tid] = z0[above];
  P[2 * CG_RUN + tid] = z0[below];
  if (end >= 0) P[end_at] = z0[end];
  if (mine) {
    P[CG_RUN + 1 + tid] = z0[n];
    r = r0[n];
    d = dinv[n];
#pragma unroll 12
    for (int q = 0; q < 36; ++q) Js[q * NTF + tid] = J[(size_t)q * N + n];
  }
  double rz = cg->rz, pq = 0.0, alpha = 0.0, beta = 0.0, rr = cg->rr;
  const double tol = cg->rtol * cg->rtol * cg->bb;
  const int maxit = cg->maxit;
  int its = 0, done = cg->done;
  // a node with three neighbours outside the runs (no grid has one): the solve gives up at once
  if (__syncthreads_or(lone)) done = 4;
  while (!done) {
    const unsigned round = (unsigned)its + 1u;
    double2 y = make_double2(0.0, 0.0), pn = y;
    double acc[1] = {0.0};
    if (mine) {
      pn = P[CG_RUN + 1 + tid];
#pragma unroll
      for (int b = 0; b < 9; ++b) {
        const double2 pb = b == 4 ? pn : (at[b] >= 0 ? P[at[b]] : at[b] == -1 ? pa : pa2);
        y.x += two(Js[(b * 4 + 0) * NTF + tid], pb.x, Js[(b * 4 + 1) * NTF + tid], pb.y);
        y.y += two(Js[(b * 4 + 2) * NTF + tid], pb.x, Js[(b * 4 + 3) * NTF + tid], pb.y);
      }
      acc[0] += dot(pn, y);
    }
    double tq[1];
    if (!exchange_sum<1>(acc, slots_q, round, tq)) {
      done = 4;
      break;
    }
    pq = tq[0];
    if (!(pq > 0.0)) {   // J not positive definite along p
      done = 2;
      break;
    }
    alpha = rz / pq;
    double acc2[2] = {0.0, 0.0};
    if (mine) {
      x = axpy(alpha, pn, x);
      r = axpy(-alpha, y, r);
      z = bmul(d, r);
      // every owner has posted its (p, q) of this round, so none still reads the last round's z
      zex.put(n, z, round);
      acc2[0] += dot(r, z);
      acc2[1] += dot(r, r);
    }
    double tr[2];
    if (!exchange_sum<2>(acc2, slots_r, round, tr)) {
      done = 4;
      break;
    }
    beta = tr[0] / rz;
    rz = tr[0];
    rr = tr[1];
    its += 1;
    if (rr <= tol) done = 1;
    else if (its >= maxit) done = 3;
    if (done) break;
    // read after the sums, when the words are there: reads before them, repeated by every thread
    // until the owners have written, hold the sums up
    auto direction = [&](const double2 &zn, const double2 &p) { return axpy(beta, p, zn); };
    bool ok;
    if (more) {   // warps that also read rows' ends or runs' ends
      const int nodes[5] = {above, below, apart[0] >= 0 ? apart[0] : above, apart[1] >= 0 ? apart[1] : above,
                            end >= 0 ? end : above};
      double2 v[5];
      ok = zex.template get<5>(nodes, round, v);
      P[tid] = direction(v[0], P[tid]);
      P[2 * CG_RUN + tid] = direction(v[1], P[2 * CG_RUN + tid]);
      pa = direction(v[2], pa);
      pa2 = direction(v[3], pa2);
      if (end >= 0) P[end_at] = direction(v[4], P[end_at]);
    } else {
      const int nodes[2] = {above, below};
      double2 v[2];
      ok = zex.template get<2>(nodes, round, v);
      P[tid] = direction(v[0], P[tid]);
      P[2 * CG_RUN + tid] = direction(v[1], P[2 * CG_RUN + tid]);
    }
    if (mine) P[CG_RUN + 1 + tid] = direction(z, pn);
    if (__syncthreads_or(!ok)) done = 4;   // its next sum is never posted: the other blocks give up too
  }
  if (mine) x_out[n] = x;
  if (blockIdx.x == 0 && tid == 0) {
    cg->rz = rz;
    cg->pq = pq;
    cg->rr = rr;
    cg->alpha = alpha;
    cg->beta = beta;
    cg->its = its;
    cg->done = done;
  }
}

// trial = vel + lambda du, with ||lambda du||^2 and ||trial||^2
__global__ void __launch_bounds__(NTF) k_fem_trial(int N, const double2 *vel, const double2 *du, double lambda,
                                                   double2 *trial, FemScalars *sc, double *partials,
                                                   unsigned *ticket) {
  double acc[2] = {0.0, 0.0};
  for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < N; n += gridDim.x * blockDim.x) {
    const double2 s = make_double2(lambda * du[n].x, lambda * du[n].y), v = vel[n];
    const double2 t = make_double2(v.x + s.x, v.y + s.y);
    trial[n] = t;
    acc[0] += s.x * s.x + s.y * s.y;
    acc[1] += t.x * t.x + t.y * t.y;
  }
  double tot[2];
  if (grid_reduce<2>(acc, partials, ticket, tot)) {
    sc->step2 = tot[0];
    sc->x2 = tot[1];
  }
}

FemGrid fem_grid(const FemProblem &P) {
  FemGrid G;
  G.Mx = P.Mx;
  G.My = P.My;
  G.px = (P.periodicity & 1) ? 1 : 0;
  G.py = (P.periodicity & 2) ? 1 : 0;
  G.nex = G.px ? P.Mx : P.Mx - 1;   // ElementMap, FETools.cc:38-83
  G.ney = G.py ? P.My : P.My - 1;
  return G;
}

int blocks(const Launch &L, int n) { return std::max(1, std::min((n + NTF - 1) / NTF, L.max_blocks)); }

template <typename T>
int alloc(T **p, size_t count) {
  return cudaMalloc((void **)p, sizeof(T) * std::max<size_t>(count, 1)) == cudaSuccess ? 0 : 1;
}

}  // namespace

FemGerms fem_germs(double dx, double dy) {
  // ShapeQ1 (FETools.hh:187-213) at the Gauss points (FETools.cc:512-519)
  const double g = 0.57735026918962573;
  const double qp[4][2] = {{-g, -g}, {g, -g}, {g, g}, {-g, g}};
  const double jx = 0.5 * dx, jy = 0.5 * dy;
  FemGerms W;
  for (int q = 0; q < 4; ++q) {
    const double x = qp[q][0], y = qp[q][1];
    const double v[4] = {(1 - x) * (1 - y) / 4., (1 + x) * (1 - y) / 4., (1 + x) * (1 + y) / 4.,
                         (1 - x) * (1 + y) / 4.};
    const double ddx[4] = {-(1 - y) / 4., (1 - y) / 4., (1 + y) / 4., -(1 + y) / 4.};
    const double ddy[4] = {-(1 - x) / 4, -(1 + x) / 4, (1 + x) / 4, (1 - x) / 4};
    for (int k = 0; k < 4; ++k) {
      W.val[q][k] = v[k];
      W.gx[q][k] = ddx[k] / jx;
      W.gy[q][k] = ddy[k] / jy;
    }
    W.JxW[q] = jx * jy * 1.0;
  }
  return W;
}

int fem_allocate(FemState &S, int Mx, int My, int periodicity) {
  const int nex = (periodicity & 1) ? Mx : Mx - 1, ney = (periodicity & 2) ? My : My - 1;
  if (S.J && S.N == Mx * My && S.nex == nex && S.ney == ney) return 0;
  fem_free(S);
  S.nex = nex;
  S.ney = ney;
  S.Ne = nex * ney;
  S.N = Mx * My;
  const size_t Q = 4 * (size_t)S.Ne, N = S.N;
  int bad = alloc(&S.C.H, Q) | alloc(&S.C.tauc, Q) | alloc(&S.C.tdu, Q) | alloc(&S.C.tdv, Q) | alloc(&S.C.B, Q) |
            alloc(&S.C.mask, Q) | alloc(&S.J, 36 * N) | alloc(&S.dinv, N) | alloc(&S.F, N) | alloc(&S.Ft, N) |
            alloc(&S.du, N) | alloc(&S.trial, N) | alloc(&S.vel0, N) | alloc(&S.r, N) | alloc(&S.z, N) | alloc(&S.p, N) |
            alloc(&S.q, N) | alloc(&S.cg, 1) | alloc(&S.sc, 1) | alloc(&S.zero_pivot, 1);
  if (bad) {
    fem_free(S);
    return 1;
  }
  return 0;
}

void fem_free(FemState &S) {
  void *ptrs[] = {S.C.H, S.C.tauc, S.C.tdu, S.C.tdv, S.C.B, S.C.mask, S.J, S.dinv, S.F, S.Ft,
                  S.du, S.trial, S.vel0, S.r, S.z, S.p, S.q, S.cg, S.sc, S.zero_pivot, S.ex};
  for (void *p : ptrs)
    if (p) cudaFree(p);
  if (S.cg_batch) cudaGraphExecDestroy(S.cg_batch);
  S = FemState{};
}

void launch_fem_coefficients(const Launch &L, const FemProblem &P, const FemState &S, const double *H,
                             const double *bed, const double *tauc, const double *srf, const double *enthalpy,
                             const double *z, int Mz, double icefree_thickness, double is_floating_thickness) {
  const FemGrid G = fem_grid(P);
  L.tick();
  k_fem_coefficients<<<blocks(L, S.Ne), NTF, 0, L.stream>>>(G, P.c, P.W, S.C, H, bed, tauc, srf, enthalpy, z, Mz,
                                                            icefree_thickness, is_floating_thickness);
}

void launch_fem_residual(const Launch &L, const FemProblem &P, const FemState &S, const double2 *vel, double2 *F,
                         bool jacobian, const uint8_t *bc, const double2 *bcv) {
  const FemGrid G = fem_grid(P);
  L.tick();
  if (jacobian)
    k_fem_node<true><<<blocks(L, S.N), NTF, 0, L.stream>>>(P, G, S.C, vel, bc, bcv, F, S.J, S.dinv, S.zero_pivot,
                                                           S.sc, L.partials, L.ticket);
  else
    k_fem_node<false><<<blocks(L, S.N), NTF, 0, L.stream>>>(P, G, S.C, vel, bc, bcv, F, S.J, S.dinv,
                                                            S.zero_pivot, S.sc, L.partials, L.ticket);
}

void launch_fem_cg_init(const Launch &L, const FemProblem &P, const FemState &S, double rtol, int maxit) {
  L.tick();
  k_cg_init<<<blocks(L, S.N), NTF, 0, L.stream>>>(S.N, S.F, S.dinv, S.du, S.r, S.z, S.p, S.cg, rtol, maxit,
                                                  L.partials, L.ticket);
  (void)P;
}

void launch_fem_cg_iterations(const Launch &L, const FemProblem &P, const FemState &S, int n) {
  const FemGrid G = fem_grid(P);
  const int b = blocks(L, S.N);
  for (int it = 0; it < n; ++it) {
    L.tick(3);
    k_cg_apply<<<b, NTF, 0, L.stream>>>(G, S.J, S.p, S.q, S.cg, L.partials, L.ticket);
    k_cg_update<<<b, NTF, 0, L.stream>>>(S.N, S.dinv, S.p, S.q, S.du, S.r, S.z, S.cg, L.partials, L.ticket);
    k_cg_direction<<<b, NTF, 0, L.stream>>>(S.N, S.z, S.p, S.cg);
  }
}

template <class Limit>
static cudaError_t run_cg_resident(const Launch &L, FemGrid G, FemState &S, int nb, Limit limit) {
  const size_t ws = ex_slot_words(nb);
  ExSlots<Limit> sq{S.ex, limit}, sr{S.ex + ws, limit};
  ExNodes<Limit> zex{S.ex + 2 * ws, S.N, limit};
  const double *J = S.J;
  const double4 *dinv = S.dinv;
  const double2 *r = S.r, *z = S.z;
  void *args[] = {&G, &J, &dinv, &r, &z, &S.du, &zex, &S.cg, &sq, &sr};
  return cudaLaunchCooperativeKernel((const void *)k_cg_resident<Limit>, dim3(nb), dim3(NTF), args, CG_SMEM, L.stream);
}

bool launch_fem_cg_resident(const Launch &L, const FemProblem &P, FemState &S) {
  const int nb = (S.N + NTF - 1) / NTF;
  if (!S.cg_resident_blocks) {   // once per grid: what the device holds at once
    S.cg_resident_blocks = INT_MAX;
    for (const void *k : {(const void *)k_cg_resident<ExDefaultLimit>, (const void *)k_cg_resident<ExGivenLimit>}) {
      cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, CG_SMEM);
      S.cg_resident_blocks = std::min(S.cg_resident_blocks, std::max(1, resident_blocks(k, NTF, CG_SMEM)));
    }
  }
  // one thread a node: the order of the sums is that of the kernels below L.max_blocks blocks
  if (nb > S.cg_resident_blocks || nb > L.max_blocks) return false;
  const size_t ws = ex_slot_words(nb), words = 2 * ws + ex_node_words(S.N);   // the slots, then z by node
  if (!S.ex && alloc(&S.ex, words) != 0) {
    cudaGetLastError();
    return false;
  }
  if (cudaMemsetAsync(S.ex, 0, sizeof(unsigned long long) * words, L.stream) != cudaSuccess) return false;
  const cudaError_t e = L.wait_limit == EX_SPIN_LIMIT ? run_cg_resident(L, fem_grid(P), S, nb, ExDefaultLimit{})
                                                      : run_cg_resident(L, fem_grid(P), S, nb, ExGivenLimit{L.wait_limit});
  if (e != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  L.tick();
  return true;
}

void launch_fem_trial(const Launch &L, const FemState &S, const double2 *vel, double lambda) {
  L.tick();
  k_fem_trial<<<blocks(L, S.N), NTF, 0, L.stream>>>(S.N, vel, S.du, lambda, S.trial, S.sc, L.partials, L.ticket);
}

}  // namespace pism_gpu
