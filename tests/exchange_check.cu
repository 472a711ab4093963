// The exchange of ssa_exchange.cuh by itself, with a block that never posts: reads lines
//   <blocks> <absent block, -1 for none> <read limit> <0: two values, 1: one value>
// runs ROUNDS sums of known values in one cooperative kernel (an absent block returns at once; a
// block whose sum fails stops there), and prints for each line how many blocks finished each
// round, and whether every sum that a block took for complete was the right one.  The words are
// zeroed and every wait is bounded, so each run ends.
#include <cstdio>
#include <vector>

#include "ssa_exchange.cuh"

using namespace pism_gpu;

constexpr int ROUNDS = 3;

__device__ double value_of(int block, int thread, int v, unsigned round) {
  return (double)((block + 1) * (v + 1) * (int)round + thread);   // whole numbers: every order adds alike
}

template <int NV, class Limit>
__global__ void __launch_bounds__(RED_THREADS) k_check(ExSlots<Limit> a, ExSlots<Limit> b, int absent, int *rounds, double *sums) {
  if ((int)blockIdx.x == absent) return;
  for (unsigned round = 1; round <= ROUNDS; ++round) {
    double x[NV], tot[NV];
    for (int v = 0; v < NV; ++v) x[v] = value_of(blockIdx.x, threadIdx.x, v, round);
    if (!exchange_sum<NV>(x, round & 1 ? a : b, round, tot)) return;
    if (threadIdx.x == 0) {
      rounds[blockIdx.x] = (int)round;
      for (int v = 0; v < NV; ++v) sums[(blockIdx.x * ROUNDS + round - 1) * 2 + v] = tot[v];
    }
  }
}

template <int NV, class Limit>
static int run(int blocks, int absent, Limit limit) {
  const size_t words = ex_slot_words(blocks);
  unsigned long long *w = nullptr;
  int *rounds = nullptr;
  double *sums = nullptr;
  if (cudaMallocManaged(&w, 2 * words * sizeof(*w)) != cudaSuccess ||
      cudaMallocManaged(&rounds, blocks * sizeof(int)) != cudaSuccess ||
      cudaMallocManaged(&sums, blocks * ROUNDS * 2 * sizeof(double)) != cudaSuccess)
    return 1;
  cudaMemset(w, 0, 2 * words * sizeof(*w));
  cudaMemset(rounds, 0, blocks * sizeof(int));
  ExSlots<Limit> a{w, limit}, b{w + words, limit};
  void *args[] = {&a, &b, &absent, &rounds, &sums};
  const void *kernel = (const void *)k_check<NV, Limit>;
  if (blocks > resident_blocks(kernel, RED_THREADS, 0) ||
      cudaLaunchCooperativeKernel(kernel, dim3(blocks), dim3(RED_THREADS), args, 0, 0) != cudaSuccess ||
      cudaDeviceSynchronize() != cudaSuccess)
    return 1;
  int done[ROUNDS] = {}, right = 1;
  for (int q = 0; q < blocks; ++q)
    for (int r = 0; r < rounds[q]; ++r) {
      done[r] += 1;
      for (int v = 0; v < NV; ++v) {
        double want = 0.0;
        for (int p = 0; p < blocks; ++p)
          for (int t = 0; t < RED_THREADS; ++t) want += (double)((p + 1) * (v + 1) * (r + 1) + t);
        if (sums[(q * ROUNDS + r) * 2 + v] != want) right = 0;
      }
    }
  for (int r = 0; r < ROUNDS; ++r) printf("%d ", done[r]);
  printf("%d\n", right);
  fflush(stdout);
  cudaFree(w);
  cudaFree(rounds);
  cudaFree(sums);
  return 0;
}

int main() {
  int blocks, absent, limit, one;
  while (scanf("%d %d %d %d", &blocks, &absent, &limit, &one) == 4)
    if (limit == EX_SPIN_LIMIT ? (one ? run<1>(blocks, absent, ExDefaultLimit{}) : run<2>(blocks, absent, ExDefaultLimit{}))
                               : (one ? run<1>(blocks, absent, ExGivenLimit{limit}) : run<2>(blocks, absent, ExGivenLimit{limit})))
      return 1;
  return 0;
}
