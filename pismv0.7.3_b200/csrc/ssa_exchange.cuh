// ssa_exchange.cuh — grid-wide sums and halo values inside one cooperative kernel, for Krylov
// solves whose data stay on chip between iterations.
//
// Every block posts its partial sums in a slot of its own; a slot's 64-bit words carry the
// round's number beside 32 bits of a value each, so a reader that finds the number in every
// word has the values too: posting, arriving and broadcasting are one trip through L2, without
// fences and without a counter that all blocks update.  Grids of more than 32 blocks add the
// slots in two trips (one warp of a leading block per 32 blocks posts their sum, then every block
// reads the at most eight sums), because every block reading every slot floods L2: 227 blocks
// took 3.3 us a sum that way and 10.9 us with fences around the halo's plain values.  The partial
// sums are added in the order of ssa_reduce.cuh, by every block alike, so all take the same
// decisions.
//
// The blocks wait for one another: the kernel is launched cooperatively, with no more blocks
// than are resident at once, and every wait gives up after a bounded number of reads.  A block that
// gives up posts nothing more, a leading block no sum of a part it has not seen whole, so no block
// takes a sum with a part missing for a sum: the others run out of reads in their turn.
#pragma once

#include "ssa_reduce.cuh"

namespace pism_gpu {

// How many reads of a word a wait takes before it gives up: the default, known to the compiler, or a
// caller's.  With every wait on a number it does not know, the resident conjugate gradients on 241^2
// nodes (227 blocks, two an SM) took 2.1 ms in place of 1.3, so a kernel has both forms.
struct ExDefaultLimit {
  static __device__ __forceinline__ constexpr int reads() { return EX_SPIN_LIMIT; }
};
struct ExGivenLimit {
  int n;
  __device__ __forceinline__ int reads() const { return n; }
};

constexpr int EX_WORDS = 4;              // a slot: two values, 32 bytes
constexpr int EX_GROUPS = RED_THREADS / 32;

// The slots of one kind of exchange: one per block, then EX_GROUPS for the leading blocks' sums.
// Kinds alternate within an iteration, so that a block may post the next round's before another
// has read this one's.  Zeroed before the kernel; rounds count from 1.
template <class Limit>
struct ExSlots {
  unsigned long long *w;
  Limit limit;
  __device__ __forceinline__ unsigned long long *block(int b) const { return w + (size_t)b * EX_WORDS; }
  __device__ __forceinline__ unsigned long long *group(int g) const { return w + (size_t)(gridDim.x + g) * EX_WORDS; }
};
inline size_t ex_slot_words(int blocks) { return (size_t)(blocks + EX_GROUPS) * EX_WORDS; }

// a double in two tagged words
__device__ __forceinline__ void ex_put(unsigned long long *p, double v, unsigned round) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"((bits & 0xffffffff00000000ull) | round),
               "l"((bits << 32) | round)
               : "memory");
}
// the NV doubles of a slot, their loads in flight together; false when the wait gave up
template <int NV, class Limit>
__device__ __forceinline__ bool ex_get(const unsigned long long *p, unsigned round, Limit limit, double (&v)[NV]) {
  for (int it = 0; it < limit.reads(); ++it) {
    unsigned long long w[NV][2];
#pragma unroll
    for (int k = 0; k < NV; ++k)
      asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                   : "=l"(w[k][0]), "=l"(w[k][1])
                   : "l"(p + 2 * k)
                   : "memory");
    bool all = true;
#pragma unroll
    for (int k = 0; k < NV; ++k) all = all && (unsigned)w[k][0] == round && (unsigned)w[k][1] == round;
    if (all) {
#pragma unroll
      for (int k = 0; k < NV; ++k)
        v[k] = __longlong_as_double((long long)((w[k][0] & 0xffffffff00000000ull) | (w[k][1] >> 32)));
      return true;
    }
  }
  return false;
}

// Vector values (two doubles) by node, in two planes of tagged words, so that a warp's nodes are
// whole sectors: the components of node n at w[2 n] and w[2 (nodes + n)].
template <class Limit>
struct ExNodes {
  unsigned long long *w;
  int nodes;
  Limit limit;
  __device__ __forceinline__ void put(int n, const double2 &v, unsigned round) const {
    ex_put(w + 2 * (size_t)n, v.x, round);
    ex_put(w + 2 * ((size_t)nodes + n), v.y, round);
  }
  // the values of M nodes, their loads in flight together; false when the wait gave up
  template <int M>
  __device__ __forceinline__ bool get(const int (&n)[M], unsigned round, double2 (&v)[M]) const {
    for (int it = 0; it < limit.reads(); ++it) {
      unsigned long long q[M][4];
#pragma unroll
      for (int m = 0; m < M; ++m)
#pragma unroll
        for (int c = 0; c < 2; ++c)
          asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                       : "=l"(q[m][2 * c]), "=l"(q[m][2 * c + 1])
                       : "l"(w + 2 * ((size_t)c * nodes + n[m]))
                       : "memory");
      bool all = true;
#pragma unroll
      for (int m = 0; m < M; ++m)
#pragma unroll
        for (int k = 0; k < 4; ++k) all = all && (unsigned)q[m][k] == round;
      if (all) {
#pragma unroll
        for (int m = 0; m < M; ++m)
          v[m] = make_double2(
              __longlong_as_double((long long)((q[m][0] & 0xffffffff00000000ull) | (q[m][1] >> 32))),
              __longlong_as_double((long long)((q[m][2] & 0xffffffff00000000ull) | (q[m][3] >> 32))));
        return true;
      }
    }
    return false;
  }
};
inline size_t ex_node_words(int nodes) { return 4 * (size_t)nodes; }

// Sum NV values over the first nb blocks of the grid; every thread of the grid gets the totals.
// False (in every thread of the block) when a wait gave up; the other blocks then give up too.
template <int NV, class Limit>
__device__ __forceinline__ bool exchange_sum(double (&val)[NV], const ExSlots<Limit> &slots, unsigned round,
                                             double (&tot)[NV], int nb = gridDim.x) {
  static_assert(2 * NV <= EX_WORDS, "a slot holds two values");
  constexpr int WARPS = RED_THREADS / 32;
  __shared__ double part[NV][WARPS], total[NV];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const double s = warp_sum(val[v]);
    if (lane == 0) part[v][warp] = s;
  }
  __syncthreads();
  bool ok = true;
  if (threadIdx.x < NV && (int)blockIdx.x < nb) {
    double s = 0.0;
    for (int q = 0; q < WARPS; ++q) s += part[threadIdx.x][q];
    ex_put(slots.block(blockIdx.x) + 2 * threadIdx.x, s, round);
  }
  // the sum of slots 32 g + lane (and those RED_THREADS further), as warp g of ssa_reduce.cuh adds it
  auto gather = [&](int g, double (&acc)[NV]) {
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = 0.0;
    for (int b = 32 * g + lane; b < nb; b += RED_THREADS) {
      double x[NV] = {};
      ok = ex_get<NV>(slots.block(b), round, slots.limit, x) && ok;
#pragma unroll
      for (int v = 0; v < NV; ++v) acc[v] += x[v];
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) acc[v] = warp_sum(acc[v]);
  };
  if (nb <= 32) {
    if (warp == 0) {
      double acc[NV];
      gather(0, acc);
#pragma unroll
      for (int v = 0; v < NV; ++v)
        if (lane == 0) total[v] = 0.0 + acc[v];
    }
  } else {
    const int groups = nb < RED_THREADS ? (nb + 31) / 32 : EX_GROUPS;
    if (warp == 1 && (int)blockIdx.x < groups) {
      double acc[NV];
      gather(blockIdx.x, acc);
      if (__all_sync(0xffffffffu, ok)) {   // else a slot is missing, and its zero is in the sum
#pragma unroll
        for (int v = 0; v < NV; ++v)
          if (lane == v) ex_put(slots.group(blockIdx.x) + 2 * v, acc[v], round);
      }
    }
    if (warp == 0) {
      double x[NV] = {};
      if (lane < groups) ok = ex_get<NV>(slots.group(lane), round, slots.limit, x) && ok;
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        double s = 0.0;
        for (int q = 0; q < groups; ++q) s += __shfl_sync(0xffffffffu, x[v], q);
        if (lane == 0) total[v] = s;
      }
    }
  }
  if (__syncthreads_or(!ok)) return false;
#pragma unroll
  for (int v = 0; v < NV; ++v) tot[v] = total[v];
  return true;
}

// how many blocks of a cooperative kernel the device holds at once (0 when the query fails)
inline int resident_blocks(const void *kernel, int threads, size_t smem) {
  int dev = 0, sms = 0, per_sm = 0, coop = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return sms * per_sm;
}

}  // namespace pism_gpu
