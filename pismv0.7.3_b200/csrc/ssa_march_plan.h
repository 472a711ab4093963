// ssa_march_plan.h — how the marching fine-level passes (ssa_march.cuh) divide a grid (host).
#pragma once

namespace pism_gpu {

constexpr int MARCH_WARPS = 4;

// strips of W = 32 - 2 halo columns, chunks of R rows; one strip's chunk is one warp's work
struct MarchPlan {
  int strips, R, chunks, blocks;
};

// All warps are resident at once (k blocks of four warps on each SM), so a pass takes R + extra
// rows, each of latency + k issue (relative units, fitted to the passes' times at 801^2 with k
// = 1 .. 4: 26.9, 14.0, 11.2, 9.0 us for the restriction, 45.7, 27.8, 21.3, 17.4 us for the
// smoothing with the apply).  A row is a chain of about 200 - 300 dependent instructions, so
// more warps cost a row little and shorten the chunks: k is 4 but on small grids, where R is
// already at its least.  A grid with more strips than that many warps takes a chunk a strip, in
// more than one wave of blocks.
inline MarchPlan march_plan(int Mx, int My, int halo, int extra, int align, int sms, int latency, int issue) {
  const int W = 32 - 2 * halo;
  MarchPlan best{};
  long long least = -1;
  for (int k = 1; k <= 4; ++k) {
    MarchPlan p;
    p.strips = (My + W - 1) / W;
    const int most = k * sms * MARCH_WARPS / p.strips;   // chunks that fit in one wave
    if (most < 1 && k < 4) continue;
    const int chunks = most < 1 ? 1 : (most < Mx ? most : Mx);
    p.R = ((Mx + chunks - 1) / chunks + align - 1) / align * align;
    p.chunks = (Mx + p.R - 1) / p.R;
    p.blocks = (p.strips * p.chunks + MARCH_WARPS - 1) / MARCH_WARPS;
    const long long cost = (p.R + extra) * (long long)(latency + k * issue);
    if (least < 0 || cost < least) {
      least = cost;
      best = p;
    }
  }
  return best;
}

// the smoothing with the operator apply, whose epilogue adds up to two sums over its blocks
inline MarchPlan march_plan_apply(int Mx, int My, int sms) { return march_plan(Mx, My, 2, 4, 1, sms, 16, 1); }

// the partial sums (doubles) it writes: its blocks have no bound in the SMs, so what holds the
// sums of the other reductions (a few a resident block) need not hold these
inline long long march_partials(int Mx, int My, int sms) { return 2LL * march_plan_apply(Mx, My, sms).blocks; }

}  // namespace pism_gpu
