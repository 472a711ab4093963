// ssa_column.cu — the consumers of the SSA velocity in StressBalance::update with a full
// update (PISMStressBalance.cc:79-116), on the device, from the handle's velocity, mask,
// thickness and enthalpy columns:
//
//   u3, v3  ConstantInColumn::update (SSB_Modifier.cc:126-152): every level of the 3-D
//           horizontal velocity is the column's SSA velocity
//   sigma   StressBalance::compute_volumetric_strain_heating (PISMStressBalance.cc:369-499)
//   w3      StressBalance::compute_vertical_velocity (PISMStressBalance.cc:192-287)
//
// The 3-D fields are [i][j][k] (a column's Mz levels contiguous).  One thread per column:
// the horizontal velocity is constant in each column, so u_z = v_z = 0 exactly and the
// horizontal derivatives, D^2 and its power are the column's, computed once; the thread then
// walks up its column, scaling the strain heating by each level's hardness and summing w by the
// trapezoid rule in the reference's order of operations.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <map>
#include <mutex>

#include "ssa_internal.h"

namespace pism_gpu {

namespace {

constexpr int NTC = 128;   // small blocks: more of the tiles fit an SM

__device__ __forceinline__ bool icy(int m) { return m == 2 || m == 3; }   // Mask.hh:46-48

// the margin-aware difference weights of one column (PISMStressBalance.cc:229-257): (west,
// east, D_x), (south, north, D_y)
struct ColumnDiff {
  double west, east, D_x, south, north, D_y;
};

__device__ __forceinline__ ColumnDiff column_diff(const GridDev &g, const int8_t *__restrict__ mask, int i, int j) {
  const int m = mask[cell(g, i, j)];
  auto cut = [&](int di, int dj) {
    const int n = mask[nbr(g, i, j, di, dj)];
    return ((icy(m) && !icy(n)) || (!icy(m) && icy(n))) ? 0.0 : 1.0;
  };
  ColumnDiff d;
  d.east = cut(1, 0);
  d.west = cut(-1, 0);
  d.north = cut(0, 1);
  d.south = cut(0, -1);
  d.D_x = d.east + d.west > 0 ? 1.0 / (g.dx * (d.east + d.west)) : 0.0;
  d.D_y = d.north + d.south > 0 ? 1.0 / (g.dy * (d.north + d.south)) : 0.0;
  return d;
}

// IceGrid::kBelowHeight through gsl_interp_accel_find: the largest k in [0, Mz - 2] with
// z[k] <= height (GSL's bisection, lo = 0, hi = Mz - 1)
__device__ __forceinline__ int k_below_height(const double *__restrict__ z, int Mz, double height) {
  int lo = 0, hi = Mz - 1;
  while (hi > lo + 1) {
    const int mid = (lo + hi) / 2;
    if (z[mid] > height) hi = mid;
    else lo = mid;
  }
  return lo;
}

// The hardness of the flow laws whose softness is Paterson and Budd's A exp(-Q / (R T)) with one
// exponential: with p = 1/n as rounded, (A exp(-x))^(-p) = A^(-p) exp(x p).  The exponent x p is near
// 9, so its rounding would be several of the result's: what the product loses is put back as a
// factor (exp(y + r) = exp(y) (1 + r), r below 1e-15), with what A^(-p) and the last product lose.
// `melting` is the value at the melting point.
struct ColdLaw {
  double A_cold, Q_cold, A_warm, Q_warm;   // A^(-p), Q
  double lost_cold, lost_warm;             // the relative rounding of A^(-p)
  double R, p;
  double melting;
};

__host__ __device__ inline double paterson_budd_hardness(const ColdLaw &l, bool cold, double T) {
  const double x = (cold ? l.Q_cold : l.Q_warm) / (l.R * T), y = x * l.p;
  const double r = fma(x, l.p, -y) + (cold ? l.lost_cold : l.lost_warm);
  const double A = cold ? l.A_cold : l.A_warm, e = exp(y), B = A * e;
  const double lost = fma(A, e, -B);
  return B > 0.0 && B < INFINITY ? B + fma(B, r, lost) : B;   // an exponent out of range leaves no remainder
}

// hardness_parameter() for the GPBLD and Paterson-Budd laws through ColdLaw
__device__ __forceinline__ double cold_hardness(const pism_gpu_ssa_config &c, const ColdLaw &l, double E, double P) {
  const double T = ec_pressure_adjusted_temperature(c, E, P);
  double B = paterson_budd_hardness(l, T < c.Paterson_Budd_critical_temperature, T);
  if (c.flow_law == PISM_FLOW_LAW_GPBLD && !(E < ec_enthalpy_cts(c, P))) {   // temperate: softened by its water
    const double omega = fmin(ec_water_fraction(c, E, P), c.gpbld_water_frac_observed_limit);
    B = l.melting * pow(1.0 + c.gpbld_water_frac_coeff * omega, -1.0 / c.ssa_Glen_exponent);
  }
  return B;
}

// One warp per 32 consecutive columns (whose [i][j][k] data are 32 Mz consecutive doubles).  The
// horizontal velocity goes out with consecutive lanes on consecutive addresses, the column's value
// taken from its lane.  The strain heating and w are computed column by column (lane r: column
// c0 + r) in a shared-memory tile, rows padded to an odd length so that the lanes' accesses at one
// level fall in different banks: the enthalpy is copied in while the velocity goes out (levels in
// the ice only), the heating takes its place, and the tile is copied out in address order.  pairs:
// two elements a lane at a time (every array 16-byte aligned).
//
// Bound: memory, 1.07 GB for 801 x 801 x 41 with GPBLD (164 us at 6.5 TB/s); the FP64 exponentials
// next to it.  With 8-warp blocks, every field through the tile, enthalpy read by columns and
// pow(exp()) a level: 461 us (12 warps an SM, 0.39 instructions a cycle and scheduler, 203 M
// instructions); one element a lane 267 us (175 M), two 187 us (93 M).
template <bool COLD>
__global__ void __launch_bounds__(NTC) k_stress_balance_3d(GridDev g, pism_gpu_ssa_config c, ColdLaw law, int Mz, int S, bool pairs,
                                                           double e_to_a_power, double exponent, double B_iso,
                                                           const double2 *__restrict__ vel,
                                                           const int8_t *__restrict__ mask,
                                                           const double *__restrict__ H,
                                                           const double *__restrict__ E,
                                                           const double *__restrict__ z,
                                                           const double *__restrict__ bmr, double *__restrict__ u3,
                                                           double *__restrict__ v3, double *__restrict__ w3,
                                                           double *__restrict__ sigma) {
  extern __shared__ __align__(16) double tiles[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  double *const tile = tiles + (size_t)warp * 32 * S;
  const int N = g.Mx * g.My;
  const int c0 = (blockIdx.x * wpb + warp) * 32;
  if (c0 >= N) return;
  const int col = c0 + lane, ncol = min(32, N - c0), n = ncol * Mz;
  const bool mine = col < N;
  const int i = mine ? col / g.My : 0, j = mine ? col - i * g.My : 0;
  const double2 U = mine ? vel[col] : make_double2(0.0, 0.0);
  const double Hc = mine ? H[col] : 0.0;
  const int ks = mine && sigma ? k_below_height(z, Mz, Hc) : -1;
  // f(e, r, k) for every element e = r Mz + k of the columns, consecutive lanes on consecutive
  // elements; all lanes call f (e >= n where there is none left)
  auto elements = [&](auto f) {
    int r = lane / Mz, k = lane - r * Mz;
    for (int e0 = 0; e0 < n; e0 += 32) {
      f(e0 + lane, r, k);
      k += 32;
      while (k >= Mz) {
        k -= Mz;
        ++r;
      }
    }
  };
  // the same for pairs of elements; column of element e by a multiplication (e < 2^15: exact)
  const unsigned inv = 0xffffffffu / (unsigned)Mz + 1u;
  auto column_of = [&](int e) { return (int)__umulhi((unsigned)e, inv); };
  auto lane_of = [&](int e) { return min(column_of(e), 31); };
  // where the tile has element e, and e + 1 behind it: both are of one column where Mz is even, and
  // with an odd Mz the rows have no padding
  const bool linear = S == Mz;
  auto at = [&](int e) { return linear ? e : e + column_of(e); };
  auto flush = [&](double *dst) {
    __syncwarp();
    double *const out = dst + (size_t)c0 * Mz;
    if (pairs) {
      for (int e = 2 * lane; e + 1 < n; e += 64) {
        const int q = at(e);
        *reinterpret_cast<double2 *>(out + e) =
            linear ? *reinterpret_cast<const double2 *>(tile + q) : make_double2(tile[q], tile[q + 1]);
      }
      if ((n & 1) && lane == 0) out[n - 1] = tile[n - 1];
    } else {
      elements([&](int e, int r, int k) {
        if (e < n) out[e] = tile[r * S + k];
      });
    }
    __syncwarp();
  };
  if (sigma && E) {
    const double *const Ec = E + (size_t)c0 * Mz;
    auto copy = [&](int e, double *to) {
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(Ec + e)
                   : "memory");
    };
    if (pairs) {
      for (int e0 = 0; e0 < n; e0 += 64) {
        const int e = e0 + 2 * lane, r = lane_of(e), k = e - r * Mz;
        // a pair across two columns begins the next one's, which has ice at its base
        const int top = __shfl_sync(0xffffffffu, ks, r);
        if (!linear && e < n && k <= top) {
          copy(e, tile + at(e));
          copy(e + 1, tile + at(e) + 1);
        } else if (linear && e + 1 < n && (k <= top || k + 1 == Mz))
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(tile + e)),
                       "l"(Ec + e)
                       : "memory");
        else if (linear && e + 1 == n && k <= top)
          copy(e, tile + e);
      }
    } else {
      elements([&](int e, int r, int k) {
        const int top = __shfl_sync(0xffffffffu, ks, r & 31);
        if (e < n && k <= top) copy(e, tile + r * S + k);
      });
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  if (u3 || v3) {
    double *const u = u3 ? u3 + (size_t)c0 * Mz : nullptr, *const v = v3 ? v3 + (size_t)c0 * Mz : nullptr;
    auto of = [&](double x, int r) { return __shfl_sync(0xffffffffu, x, r); };
    if (pairs) {
      for (int e0 = 0; e0 < n; e0 += 64) {
        const int e = e0 + 2 * lane, r = lane_of(e), q = lane_of(e + 1);
        const double2 x = make_double2(of(U.x, r), of(U.x, q)), y = make_double2(of(U.y, r), of(U.y, q));
        if (e + 1 < n) {
          if (u) *reinterpret_cast<double2 *>(u + e) = x;
          if (v) *reinterpret_cast<double2 *>(v + e) = y;
        } else if (e < n) {
          if (u) u[e] = x.x;
          if (v) v[e] = y.x;
        }
      }
    } else {
      elements([&](int e, int r, int k) {
        const double x = of(U.x, r & 31), y = of(U.y, r & 31);
        if (e < n) {
          if (u) u[e] = x;
          if (v) v[e] = y;
        }
      });
    }
  }
  if (!w3 && !sigma) return;
  double u_x = 0.0, v_y = 0.0, u_y = 0.0, v_x = 0.0;
  if (mine) {
    const ColumnDiff d = column_diff(g, mask, i, j);
    const double2 Uw = vel[nbr(g, i, j, -1, 0)], Ue = vel[nbr(g, i, j, 1, 0)], Us = vel[nbr(g, i, j, 0, -1)],
                  Un = vel[nbr(g, i, j, 0, 1)];
    u_x = d.D_x * (d.west * (U.x - Uw.x) + d.east * (Ue.x - U.x));
    v_y = d.D_y * (d.south * (U.y - Us.y) + d.north * (Un.y - U.y));
    u_y = d.D_y * (d.south * (U.x - Us.x) + d.north * (Un.x - U.x));
    v_x = d.D_x * (d.west * (U.y - Uw.y) + d.east * (Ue.y - U.y));
  }
  if (sigma) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    if (mine) {
      const double a = u_x + v_y, b = u_y + v_x;   // u_z = v_z = 0
      // D2(), PISMStressBalance.cc:309-311
      const double D2 = 0.5 * (a * a + u_x * u_x + v_y * v_y + 0.5 * (b * b));
      const double two_e = 2.0 * e_to_a_power, D2e = pow(D2, exponent);
      double *const row = tile + lane * S;
#pragma unroll 2
      for (int k = 0; k <= ks; ++k) {
        double B = B_iso;
        if constexpr (COLD) B = cold_hardness(c, law, row[k], ec_pressure(c, Hc - z[k]));
        else if (E) B = hardness_parameter(c, row[k], ec_pressure(c, Hc - z[k]));
        row[k] = two_e * B * D2e;   // the reference's order: (2 e^(-1/n) B) D^(1/n + 1)
      }
      for (int k = ks + 1; k < Mz; ++k) row[k] = 0.0;
    }
    flush(sigma);
  }
  if (w3) {
    // w(0) = -bmr (or 0); w(k) = w(k-1) - (integrand(k) + integrand(k-1)) / 2 dz, the
    // integrand u_x + v_y the same at every level; the products and sums in that order
    if (mine) {
      const double integrand = __dadd_rn(u_x, v_y);
      const double half_sum = __dmul_rn(0.5, __dadd_rn(integrand, integrand));
      double w = bmr ? -bmr[col] : 0.0, below = z[0];
      double *const row = tile + lane * S;
      row[0] = w;
#pragma unroll 4
      for (int k = 1; k < Mz; ++k) {
        const double zk = z[k];
        w = __dsub_rn(w, __dmul_rn(half_sum, __dsub_rn(zk, below)));
        row[k] = w;
        below = zk;
      }
    }
    flush(w3);
  }
}

}  // namespace

int stress_balance_3d_smem(int Mz, int *warps) {
  const int S = Mz | 1;
  const int per_warp = 32 * S * (int)sizeof(double);
  *warps = std::max(1, std::min(NTC / 32, (200 * 1024) / per_warp));
  return *warps * per_warp;
}

void launch_stress_balance_3d(const Launch &L, const GridDev &g, const pism_gpu_ssa_config &c, int Mz,
                              const Fields &f, const double *z, const double *bmr, double *u3, double *v3,
                              double *w3, double *sigma) {
  const int N = g.Mx * g.My;
  int warps = 0;
  const int smem = stress_balance_3d_smem(Mz, &warps);
  const int blocks = (N + 32 * warps - 1) / (32 * warps);
  // PISMStressBalance.cc:384-387: the flow law's exponent and enhancement factor; an
  // isothermal flow law's hardness A^(-1/n) is the same at every level
  const double n = c.ssa_Glen_exponent, exponent = 0.5 * (1.0 / n + 1.0);
  const double e_to_a_power = std::pow(c.ssa_enhancement_factor, -1.0 / n);
  const bool iso = c.flow_law == PISM_FLOW_LAW_ISOTHERMAL_GLEN;
  const double B_iso = iso ? std::pow(c.ice_softness, -1.0 / n) : 0.0;
  // the laws with one exponential a level; the others as in ssa_device.cuh
  const bool cold = c.flow_law == PISM_FLOW_LAW_GPBLD || c.flow_law == PISM_FLOW_LAW_PB;
  ColdLaw law{};
  if (cold) {
    law.p = 1.0 / n;
    law.R = c.ideal_gas_constant;
    law.Q_cold = c.Paterson_Budd_Q_cold;
    law.Q_warm = c.Paterson_Budd_Q_warm;
    const auto power = [&](double A, double *rounded, double *lost) {
      const long double v = std::pow((long double)A, -(long double)law.p);
      *rounded = (double)v;
      *lost = std::isfinite(*rounded) && *rounded > 0.0 ? (double)((v - *rounded) / v) : 0.0;
    };
    power(c.Paterson_Budd_A_cold, &law.A_cold, &law.lost_cold);
    power(c.Paterson_Budd_A_warm, &law.A_warm, &law.lost_warm);
    const double Tm = c.water_melting_point_temperature;
    law.melting = paterson_budd_hardness(law, Tm < c.Paterson_Budd_critical_temperature, Tm);
  }
  // rows of an odd length: with an odd number of levels the tile is the columns' memory as it is
  const double *const E = iso ? nullptr : f.enthalpy;
  const int S = Mz | 1;
  bool pairs = true;
  for (const double *q : {(const double *)u3, (const double *)v3, (const double *)w3, (const double *)sigma, E})
    pairs = pairs && reinterpret_cast<uintptr_t>(q) % 16 == 0;
  L.tick();
  const auto kernel = cold ? k_stress_balance_3d<true> : k_stress_balance_3d<false>;
  kernel<<<blocks, 32 * warps, smem, L.stream>>>(g, c, law, Mz, S, pairs, e_to_a_power, exponent, B_iso, f.vel, f.mask, f.H, E, z,
                                                 bmr, u3, v3, w3, sigma);
}

// the kernel's dynamic shared-memory limit for Mz levels on the current device: a function
// attribute shared by every handle on that device, so it is only ever raised, under a lock
int stress_balance_3d_prepare(int Mz) {
  static std::mutex lock;
  static std::map<int, int> raised;   // device -> bytes granted
  int warps = 0, dev = 0;
  const int smem = stress_balance_3d_smem(Mz, &warps);
  if (smem <= 48 * 1024) return 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  std::lock_guard<std::mutex> guard(lock);
  auto it = raised.find(dev);
  if (it != raised.end() && smem <= it->second) return 0;
  for (const void *kernel : {(const void *)k_stress_balance_3d<true>, (const void *)k_stress_balance_3d<false>})
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess) return 1;
  raised[dev] = smem;
  return 0;
}

}  // namespace pism_gpu
