// ssa_march.cuh — the fine-level FP32 passes of the multigrid cycle, one warp marching down a
// strip of columns.
//
// A lane owns one column and walks the rows of its chunk; the three rows of a stencil are a
// window in registers, the columns either side come from the neighbouring lanes by shuffles.  No
// shared memory, no barriers, and each row of a strip is read once, with the next row's
// loads in flight while this one computes.  The lanes at a strip's ends carry its halo (one
// column a side where one stencil is applied, two where two are), and a chunk starts its halo
// rows early, so about 1.2 - 1.5 cells are visited per cell of the result.
//
// Bound: instruction latency, a row's chain of about 200 - 300 dependent instructions on at most
// four warps a scheduler (registers); L2 and DRAM are idle by comparison.  The tiles of 32 x 8
// cells that these passes were (a two-cell halo staged through shared memory: 432 and 340 items
// on 256 threads) issued 13.0 M warp instructions for the smoothing with the operator apply on
// 641 601 cells and waited at three barriers a tile.  801^2 on one B200, tiles / marching: the
// smoothing with the apply 27.3 / 17.4 us, the restriction 13.6 / 8.2 us.  Every cell takes the
// arithmetic of those passes in the same order; only the FP64 sums of the epilogues are added in
// another order.
#pragma once

#include "ssa_fine32.cuh"
#include "ssa_krylov32.cuh"
#include "ssa_march_plan.h"
#include "ssa_pdl.cuh"

namespace pism_gpu {

constexpr int MARCH_THREADS = 32 * MARCH_WARPS;

// this warp's strip and chunk
struct MarchTask {
  int J0, I0, rows;   // rows 0: nothing to do
};
__device__ __forceinline__ MarchTask march_task(const MarchPlan &m, int Mx, int W) {
  const int task = blockIdx.x * MARCH_WARPS + (threadIdx.x >> 5);
  const int chunk = task / m.strips, strip = task - chunk * m.strips;
  MarchTask t;
  t.J0 = strip * W;
  t.I0 = chunk * m.R;
  t.rows = chunk < m.chunks ? (m.R < Mx - t.I0 ? m.R : Mx - t.I0) : 0;
  return t;
}

// v as a rounded value: the compiler may not fuse the product it came from into what reads it
__device__ __forceinline__ float2 rounded(float2 v) {
  asm volatile("" : "+f"(v.x), "+f"(v.y));
  return v;
}

// omega v + corr c, the second product rounded by itself
__device__ __forceinline__ float2 march_iterate(float omega, const float2 &v, float corr, const float2 &c) {
  return make_float2(__fmaf_rn(omega, v.x, __fmul_rn(corr, c.x)), __fmaf_rn(omega, v.y, __fmul_rn(corr, c.y)));
}

// a value and its neighbours in the columns j - 1 and j + 1
struct Row3 {
  float2 s, c, n;
};
__device__ __forceinline__ float2 lane_below(const float2 &v) {
  return make_float2(__shfl_up_sync(0xffffffffu, v.x, 1), __shfl_up_sync(0xffffffffu, v.y, 1));
}
__device__ __forceinline__ float2 lane_above(const float2 &v) {
  return make_float2(__shfl_down_sync(0xffffffffu, v.x, 1), __shfl_down_sync(0xffffffffu, v.y, 1));
}
__device__ __forceinline__ Row3 row3(const float2 &v) { return Row3{lane_below(v), v, lane_above(v)}; }

// y = A x at the middle row of the window (w: i - 1, m: i, e: i + 1)
__device__ __forceinline__ float2 march_apply(const FineF &F, int i, int j, uint32_t f, float bta, float c_w, float c_e,
                                              float c_s, float c_n, const Row3 &w, const Row3 &m, const Row3 &e) {
  auto xr = [&](int di, int dj) {
    const Row3 &r = di < 0 ? w : (di > 0 ? e : m);
    return dj < 0 ? r.s : (dj > 0 ? r.n : r.c);
  };
  return fine_apply_coef(F, i, j, f, bta, c_w, c_e, c_s, c_n, xr);
}

// ---- the loads: a ring of rows per warp, filled by asynchronous copies MARCH_AHEAD rows before
// they are used.  Every lane copies its own column and reads back only that, so a row needs no
// barrier, just the copies' group to be complete. ----
constexpr int MARCH_AHEAD = 5, MARCH_RING = MARCH_AHEAD + 1;
// a row's slot: D^-1 (16 B a lane), the packed operator (16), b (16), x_1 (8)
constexpr int MARCH_D = 0, MARCH_OP = 512, MARCH_B = 1024, MARCH_XC = 1536, MARCH_SLOT = 1792;

template <int BYTES>
__device__ __forceinline__ void march_copy(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void march_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// the oldest group but MARCH_AHEAD is complete
__device__ __forceinline__ void march_ready() { asm volatile("cp.async.wait_group %0;" ::"n"(MARCH_AHEAD) : "memory"); }

// how a right-hand side accessor's row is copied and read back
template <class V>
__device__ __forceinline__ void march_copy_b(const VecAcc<V> &b, void *dst, int k) {
  march_copy<sizeof(V)>(dst, b.p + k);
}
__device__ __forceinline__ void march_copy_b(const SAcc &b, void *dst, int k) {
  march_copy<8>(dst, b.r + k);
  march_copy<8>(static_cast<float2 *>(dst) + 1, b.v + k);
}
template <class V>
__device__ __forceinline__ float2 march_read_b(const VecAcc<V> &, const void *src) {
  return to_f2(*static_cast<const V *>(src));
}
__device__ __forceinline__ float2 march_read_b(const SAcc &b, const void *src) {
  const float4 q = *static_cast<const float4 *>(src);
  return make_float2(q.x - b.al * q.z, q.y - b.al * q.w);
}

// one lane's view of the ring
struct MarchRow {
  float4 D;
  float2 b, nu, xc;
  uint32_t f;
  float bta;
};
struct MarchRing {
  unsigned char *p;   // this lane's 16-byte column of slot 0
  int lane;
  __device__ __forceinline__ void *at(int slot, int what, int bytes) const {
    return p + slot * MARCH_SLOT + what + lane * bytes;
  }
  __device__ __forceinline__ void operator_row(const FineF &F, int slot, int k) const {
    march_copy<16>(at(slot, MARCH_D, 16), F.dinv + k);
    march_copy<16>(at(slot, MARCH_OP, 16), F.op + k);
  }
  template <class BA>
  __device__ __forceinline__ void b_row(const BA &b, int slot, int k) const {
    march_copy_b(b, at(slot, MARCH_B, 16), k);
  }
  __device__ __forceinline__ void xc_row(const float2 *xc, int slot, int q) const {
    march_copy<8>(at(slot, MARCH_XC, 8), xc + q);
  }
  template <bool XC, class BA>
  __device__ __forceinline__ MarchRow read(const BA &b, int slot) const {
    MarchRow r;
    r.D = *static_cast<const float4 *>(at(slot, MARCH_D, 16));
    r.b = march_read_b(b, at(slot, MARCH_B, 16));
    if (XC) r.xc = *static_cast<const float2 *>(at(slot, MARCH_XC, 8));
    const float4 o = *static_cast<const float4 *>(at(slot, MARCH_OP, 16));
    r.nu = make_float2(o.x, o.y);
    r.bta = o.z;
    r.f = __float_as_uint(o.w);
    return r;
  }
};
__device__ __forceinline__ int march_slot(int slot) { return slot + 1 == MARCH_RING ? 0 : slot + 1; }
#define MARCH_RING_SMEM                                                                   \
  __shared__ __align__(16) unsigned char march_smem[MARCH_WARPS][MARCH_RING][MARCH_SLOT]; \
  const MarchRing ring{&march_smem[threadIdx.x >> 5][0][0], (int)(threadIdx.x & 31)}

// walks the rows of a strip: the wrapped row and this lane's cell in it
struct MarchCell {
  int i, j, k;
};
__device__ __forceinline__ MarchCell march_start(int i, int j, int Mx, int My) {
  MarchCell c;
  c.i = pmod(i, Mx);
  c.j = pmod(j, My);
  c.k = c.i * My + c.j;
  return c;
}
__device__ __forceinline__ void march_next(MarchCell &c, int Mx, int My) {
  c.k += My;
  if (++c.i == Mx) {
    c.i = 0;
    c.k = c.j;
  }
}

// b_1 = R (b - A x0), x0 = omega D^-1 b.  Before the wait: the operator of the first rows.
template <int AX, int AY, class BA>
__global__ void __launch_bounds__(MARCH_THREADS, 4) k_mg0_restrict(FineF F, BA b_in, float omega, int Myc, MarchPlan m,
                                                                   float2 *bc, const KState *st) {
  MARCH_RING_SMEM;
  const int Mx = F.g.Mx, My = F.g.My, lane = threadIdx.x & 31;
  const MarchTask t = march_task(m, Mx, 30);
  const int jc = t.J0 - 1 + lane, T = t.rows > 0 ? t.rows + 2 : 0;
  MarchCell c = march_start(t.I0 - 1, jc, Mx, My);
  {
    MarchCell q = c;
    for (int s = 0; s < MARCH_AHEAD && s < T; ++s, march_next(q, Mx, My)) ring.operator_row(F, s, q.k);
  }
  pdl_wait();
  if (st && st->done) return;
  pdl_release();
  const auto b = b_in.bind();
#pragma unroll
  for (int s = 0; s < MARCH_AHEAD; ++s) {
    if (s < T) ring.b_row(b, s, c.k);
    march_commit();
    march_next(c, Mx, My);
  }
  const bool mine = lane >= 1 && lane <= 30 && jc < My;
  Row3 xw{}, xm{};                          // x0 of rows i - 1 and i of the stencil
  float nw = 0.0f, ns = 0.0f, btm = 0.0f;   // nu*H east of row i - 1, north of (i, j - 1); beta of row i
  float2 nm{}, bm{};                        // row i: nu*H, b
  uint32_t fm = 0;
  float2 sum = make_float2(0.0f, 0.0f);
  int use = 0, fill = MARCH_AHEAD;
#pragma unroll 2
  for (int s = 0; s < T; ++s) {
    if (s + MARCH_AHEAD < T) {
      ring.operator_row(F, fill, c.k);
      ring.b_row(b, fill, c.k);
      march_next(c, Mx, My);
    }
    march_commit();
    march_ready();
    const MarchRow q = ring.read<false>(b, use);
    use = march_slot(use);
    fill = march_slot(fill);
    const float2 v = fmul4(q.D, q.b);
    const Row3 x = row3(rounded(make_float2(omega * v.x, omega * v.y)));
    if (s >= 2) {
      const int i = t.I0 + s - 2;
      float2 r = make_float2(0.0f, 0.0f);
      if (mine) {
        const float2 y = march_apply(F, i, jc, fm, btm, nw, nm.x, ns, nm.y, xw, xm, x);
        r = make_float2(bm.x - y.x, bm.y - y.y);
      }
      const bool first = AX == 1 || (i & 1) == 0;
      sum.x = first ? r.x : sum.x + r.x;
      sum.y = first ? r.y : sum.y + r.y;
      if (AY == 2) {
        const float2 n = lane_above(r);
        sum.x += n.x;
        sum.y += n.y;
      }
      if (mine && (AY == 1 || (jc & 1) == 0) && (AX == 1 || (i & 1) == 1 || i == Mx - 1))
        bc[(i / AX) * Myc + jc / AY] = sum;
    }
    xw = xm;
    xm = x;
    nw = nm.x;
    nm = q.nu;
    ns = __shfl_up_sync(0xffffffffu, q.nu.y, 1);
    bm = q.b;
    fm = q.f;
    btm = q.bta;
  }
}

// x = omega D^-1 b + s P x_1;  z = x + omega D^-1 (b - A x).  Before the wait: everything of
// the first rows but x_1 (b was written before the cycle).
template <int AX, int AY, class BA, class ZV>
__global__ void __launch_bounds__(MARCH_THREADS, 4) k_mg0_post(FineF F, BA b_in, float omega, float corr, int Myc,
                                                               const float2 *xc_, MarchPlan m, ZV *z,
                                                               const KState *st) {
  MARCH_RING_SMEM;
  const int Mx = F.g.Mx, My = F.g.My, lane = threadIdx.x & 31;
  const MarchTask t = march_task(m, Mx, 30);
  const int jc = t.J0 - 1 + lane, T = t.rows > 0 ? t.rows + 2 : 0;
  MarchCell c = march_start(t.I0 - 1, jc, Mx, My);
  const int J = c.j / AY;
  {
    MarchCell q = c;
    for (int s = 0; s < MARCH_AHEAD && s < T; ++s, march_next(q, Mx, My)) {
      ring.operator_row(F, s, q.k);
      ring.b_row(b_in, s, q.k);
    }
  }
  pdl_wait();
  if (st && st->done) return;
  pdl_release();
  const float2 *xc = after_wait(xc_);
  const auto b = b_in.bind();
#pragma unroll
  for (int s = 0; s < MARCH_AHEAD; ++s) {
    if (s < T) ring.xc_row(xc, s, (c.i / AX) * Myc + J);
    march_commit();
    march_next(c, Mx, My);
  }
  const bool mine = lane >= 1 && lane <= 30 && jc < My;
  Row3 xw{}, xm{};
  float nw = 0.0f, ns = 0.0f, btm = 0.0f;
  float2 nm{}, bm{};
  float4 Dm{};
  uint32_t fm = 0;
  int use = 0, fill = MARCH_AHEAD;
#pragma unroll 2
  for (int s = 0; s < T; ++s) {
    if (s + MARCH_AHEAD < T) {
      ring.operator_row(F, fill, c.k);
      ring.b_row(b, fill, c.k);
      ring.xc_row(xc, fill, (c.i / AX) * Myc + J);
      march_next(c, Mx, My);
    }
    march_commit();
    march_ready();
    const MarchRow q = ring.read<true>(b, use);
    use = march_slot(use);
    fill = march_slot(fill);
    const Row3 x = row3(march_iterate(omega, fmul4(q.D, q.b), corr, q.xc));
    if (s >= 2 && mine) {
      const int i = t.I0 + s - 2;
      const float2 y = march_apply(F, i, jc, fm, btm, nw, nm.x, ns, nm.y, xw, xm, x);
      const float2 d = fmul4(Dm, make_float2(bm.x - y.x, bm.y - y.y));
      z[i * My + jc] = from_f2<ZV>(make_float2(xm.c.x + omega * d.x, xm.c.y + omega * d.y));
    }
    xw = xm;
    xm = x;
    nw = nm.x;
    nm = q.nu;
    ns = __shfl_up_sync(0xffffffffu, q.nu.y, 1);
    bm = q.b;
    Dm = q.D;
    fm = q.f;
    btm = q.bta;
  }
}

// The same fused with the FP32 operator apply that follows the V-cycle in BiCGStab: z as above
// on the strip and one column and row around it (recomputed there by its own warp as well),
// stored on the strip, and y = A z handed to the epilogue.
template <int AX, int AY, class BA, class EPI>
__global__ void __launch_bounds__(MARCH_THREADS, 4) k_mg0_post_apply(FineF F, BA b_in, float omega, float corr, int Myc,
                                                                     const float2 *xc_, MarchPlan m, float2 *z_,
                                                                     EPI e) {
  MARCH_RING_SMEM;
  const int Mx = F.g.Mx, My = F.g.My, lane = threadIdx.x & 31;
  const MarchTask t = march_task(m, Mx, 28);
  const int jc = t.J0 - 2 + lane, T = t.rows > 0 ? t.rows + 4 : 0;
  MarchCell c = march_start(t.I0 - 2, jc, Mx, My);
  const int J = c.j / AY, jw = c.j;
  int iz = pmod(t.I0 - 3, Mx);   // wrapped row of the z about to be formed
  {
    MarchCell q = c;
    for (int s = 0; s < MARCH_AHEAD && s < T; ++s, march_next(q, Mx, My)) {
      ring.operator_row(F, s, q.k);
      ring.b_row(b_in, s, q.k);
    }
  }
  pdl_wait();
  if (e.st->done) return;
  pdl_release();
  e.begin();
  const float2 *xc = after_wait(xc_);
  float2 *z = after_wait(z_);
  const auto b = b_in.bind();
#pragma unroll
  for (int s = 0; s < MARCH_AHEAD; ++s) {
    if (s < T) ring.xc_row(xc, s, (c.i / AX) * Myc + J);
    march_commit();
    march_next(c, Mx, My);
  }
  const bool mine = lane >= 2 && lane <= 29 && jc < My;
  Row3 xw{}, xm{}, zw{}, zm{};
  // row i (of x's stencil): nu*H, b, D^-1, flags, beta; row i - 1 (of z's stencil)
  float nw = 0.0f, ns = 0.0f, btm = 0.0f, nww = 0.0f, nws = 0.0f, btw = 0.0f;
  float2 nm{}, bm{}, nwm{};
  float4 Dm{};
  uint32_t fm = 0, fw = 0;
  int use = 0, fill = MARCH_AHEAD;
  for (int s = 0; s < T; ++s) {
    if (s + MARCH_AHEAD < T) {
      ring.operator_row(F, fill, c.k);
      ring.b_row(b, fill, c.k);
      ring.xc_row(xc, fill, (c.i / AX) * Myc + J);
      march_next(c, Mx, My);
    }
    march_commit();
    march_ready();
    const MarchRow q = ring.read<true>(b, use);
    use = march_slot(use);
    fill = march_slot(fill);
    const Row3 x = row3(march_iterate(omega, fmul4(q.D, q.b), corr, q.xc));
    // z at row I0 + s - 3
    float2 zc = make_float2(0.0f, 0.0f);
    if (s >= 2) {
      const float2 y = march_apply(F, iz, jw, fm, btm, nw, nm.x, ns, nm.y, xw, xm, x);
      const float2 d = fmul4(Dm, make_float2(bm.x - y.x, bm.y - y.y));
      zc = rounded(make_float2(xm.c.x + omega * d.x, xm.c.y + omega * d.y));
    }
    const Row3 zr = row3(zc);
    if (s >= 4 && mine) {
      const int i = t.I0 + s - 4, k = i * My + jc;
      z[k] = zm.c;
      e.body(k, march_apply(F, i, jc, fw, btw, nww, nwm.x, nws, nwm.y, zw, zm, zr));
    }
    if (++iz == Mx) iz = 0;
    zw = zm;
    zm = zr;
    nww = nw;
    nwm = nm;
    nws = ns;
    btw = btm;
    fw = fm;
    xw = xm;
    xm = x;
    nw = nm.x;
    nm = q.nu;
    ns = __shfl_up_sync(0xffffffffu, q.nu.y, 1);
    bm = q.b;
    Dm = q.D;
    fm = q.f;
    btm = q.bta;
  }
  e.template finish<MARCH_THREADS>();
}

}  // namespace pism_gpu
