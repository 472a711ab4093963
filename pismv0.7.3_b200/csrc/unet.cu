// unet.cu — the learned warm start's network (include/pism_unet_gpu.h): a 4-level U-Net in
// BF16 with FP32 accumulation on the tensor cores (mma.sync m16n8k16, operands staged in
// shared memory and fed by ldmatrix), its backward pass and an Adam step.
//
// The convolutions are implicit GEMMs over a tile of 8 or 16 x 16 output pixels and 32 output
// channels: the patch of one 16- or 32-channel slice and its 3 x 3 weights are copied
// asynchronously one step ahead, each warp owns one or two output rows (16 pixels a row) and all
// 32 channels, K runs over taps x channels.  The backward data pass is the same kernel on
// flipped, transposed weights; every gradient is masked by its layer's ReLU by the kernel that
// makes it.  The weight gradient is a GEMM over pixels (one warp per tap) reduced
// deterministically across CTAs, on a second stream beside the data gradients.
// Every reduction (weight / bias gradients, loss) is written as per-CTA partial sums and
// summed in a fixed order, so training runs are bit-reproducible.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <string>
#include <vector>

#include "pism_unet_gpu.h"
#include "unet_internal.h"

using bf16 = __nv_bfloat16;

namespace pism_unet {

constexpr int TH = 8, TW = 16;            // pixel tile of the weight gradient; the convolution's is 8 or 16 x 16
constexpr int PH = TH + 2, PW = TW + 2;   // input patch with the 3 x 3 halo
constexpr int THREADS = 256;              // 8 warps, one or two tile rows each
constexpr int WG_THREADS = 288;           // weight gradient: 9 warps = 9 taps
constexpr int WG_MAX_CTAS = 64;           // pixel-range partial sums per weight gradient
constexpr int BIAS_MAX_CTAS = 256;        // and per bias gradient

// ---- the network ----
struct LayerDef {
  int cin, cout, level;   // level 0 = full resolution
};
constexpr int NLAYERS = 10;
constexpr LayerDef LAYERS[NLAYERS] = {
    {16, 32, 0}, {32, 32, 0}, {32, 64, 1}, {64, 64, 1}, {64, 96, 2},
    {96, 96, 2}, {96, 128, 3}, {224, 96, 2}, {160, 64, 1}, {96, 32, 0},
};
constexpr int HEAD_CIN = 32, HEAD_COUT = 2;

long long param_count() {
  long long n = 0;
  for (const LayerDef &L : LAYERS) n += 9LL * L.cout * L.cin + L.cout;
  return n + HEAD_COUT * HEAD_CIN + HEAD_COUT;
}

// ---- device helpers ----
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], const void *p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}

__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], const void *p) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}

// d += a (16x16, row) * b (16x8, col), BF16 in, FP32 accumulate
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// keep the BF16 halves of v whose counterpart in m is > 0 (the ReLU derivative)
__device__ __forceinline__ uint32_t relu_mask2(uint32_t v, uint32_t m) {
  uint32_t keep = 0;
  if (!(m & 0x8000u) && (m & 0x7fffu)) keep |= 0x0000ffffu;
  if (!(m & 0x80000000u) && (m & 0x7fff0000u)) keep |= 0xffff0000u;
  return v & keep;
}

__device__ __forceinline__ uint4 relu_mask8(uint4 v, uint4 m) {
  return make_uint4(relu_mask2(v.x, m.x), relu_mask2(v.y, m.y), relu_mask2(v.z, m.z), relu_mask2(v.w, m.w));
}

__device__ __forceinline__ void unpack8(uint4 v, float (&f)[8]) {
  const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&v);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float2 t = __bfloat1622float2(h[q]);
    f[2 * q] = t.x;
    f[2 * q + 1] = t.y;
  }
}

__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
  uint4 v;
  __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&v);
#pragma unroll
  for (int q = 0; q < 4; ++q) h[q] = __floats2bfloat162_rn(f[2 * q], f[2 * q + 1]);
  return v;
}

// 16 bytes to shared memory, zeros where `from` is outside the image; not waited for
__device__ __forceinline__ void copy16(void *to, const void *from, bool inside) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from),
               "r"(inside ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all groups but the latest N are complete
template <int N>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// A layer's input, [b, i, j, channel]: x, or the concatenation [up[b, i/2, j/2, 0:Cu], x[b, i, j, :]]
// of the decoder, read where its parts are (as an array of its own it was written and read again,
// 45 us of kernels in a 16 x 128 x 128 step).  Cu and x's C are
// multiples of the kernels' channel slices, so a slice is in one of them.
struct ConvIn {
  const bf16 *x, *up;
  int C, Cu;
  __host__ __device__ int channels() const { return C + Cu; }
};

// Copy the ROWS x (TW+2) patch of channels [c0, c0 + CS) around the tile at (i0, j0) of image b;
// zero outside the image.
template <int CS, int NTHR, int ROWS>
__device__ __forceinline__ void copy_patch(bf16 *patch, const ConvIn &in, int c0, int b, int i0, int j0, int H, int W) {
  constexpr int CP = CS + 8, CH = CS / 8;
  const int half = c0 < in.Cu ? 1 : 0, C = half ? in.Cu : in.C, Hs = H >> half, Ws = W >> half;
  const bf16 *__restrict__ const x = half ? in.up + c0 : in.x + (c0 - in.Cu);
  for (int q = threadIdx.x; q < ROWS * PW * CH; q += NTHR) {
    const int pix = q / CH, ch = q - pix * CH;
    const int pi = pix / PW, pj = pix - pi * PW;
    const int ii = i0 - 1 + pi, jj = j0 - 1 + pj;
    const bool inside = ii >= 0 && ii < H && jj >= 0 && jj < W;
    copy16(patch + pix * CP + ch * 8, inside ? x + (((size_t)b * Hs + (ii >> half)) * Ws + (jj >> half)) * C + ch * 8 : x,
           inside);
  }
}

// ---- 3x3 convolution (forward, and backward data on flipped weights) ----
// y[b, i, j, co] = act(bias[co] + sum_{tap, ci} w[tap, co, ci] * x[b, i + ky - 1, j + kx - 1, ci]),
// zero where omask[b, i, j, co] <= 0 (backward data: the ReLU of the layer that made the input).
//
// With QUADS (and MR = 2: a warp has both rows of a 2 x 2 block, the columns are four lanes apart)
// the kernel also makes the sums over 2 x 2 blocks that follow it, of the outputs as rounded: the
// mean that the next level reads, or the gradient of the upsampled part of a concatenation; the
// gradient of its other part goes out in place.  As kernels of their own these read and wrote every
// output again: 16 x 128 x 128, convolutions with concatenations and sums 600 us of kernel time a
// step, in one 547; the step 1055 -> 988 us, the forward of 1 x 408 x 408 267 -> 235 us.
//
// A CTA walks pixel tiles of 8 MR x 16 pixels for NB output channels; each warp has MR rows (16
// pixels a row) by all NB channels.  A step is one channel slice of a tile: its patch (and its
// weights, unless the layer has one slice: then they stay) is copied asynchronously while the
// step before multiplies.
//
// Bound: the legacy tensor pipe and the loads that feed it.  Unpipelined, at 8 x 16 pixels by 32
// channels, the warps waited on global loads (9 of 17 stalled warps an issue, the tensor pipe
// 28 - 36 % active).  Every output adds the same products in the same order (slices, taps, halves
// of a slice) whatever the tile, so the tile may follow the shape.  Forward of 1 x 408 x 408 (34
// GFLOP): 314 us then, 269 us with the copies ahead.
// What a kernel with QUADS adds: q[b, I, J, co] = scale x the sum of the outputs co < C over the
// 2 x 2 block, zero where mask[b, I, J, co] <= 0; y gets the channels from y0 on, as its own
// channels 0 and up.  C and y0 are multiples of 32.
struct Quads {
  bf16 *q;
  const bf16 *mask;
  int C, y0;
  float scale;
};

template <int CS, int NB, int MR, bool RESIDENT>
constexpr int conv_smem() {
  return (2 * (8 * MR + 2) * PW + (RESIDENT ? 1 : 2) * 9 * NB) * (CS + 8) * (int)sizeof(bf16);
}

// As many CTAs an SM as the shared memory takes, at most three, and registers for them: unbounded, the
// layers whose weights stay took 93 - 96, two CTAs of the three that their grid counts on, so a
// second wave of long CTAs (32 to 96 channels of 16 x 128 x 128: 75 us, bounded 63); those with
// several slices now use up to 120 registers.
template <int CS, int NB, int MR, bool RESIDENT>
constexpr int conv_ctas() {
  return conv_smem<CS, NB, MR, RESIDENT>() * 3 <= 220 * 1024 ? 3 : 2;
}

template <int CS, int NB, int MR, bool RESIDENT, bool QUADS>
__global__ void __launch_bounds__(THREADS, (conv_ctas<CS, NB, MR, RESIDENT>())) k_conv3x3(ConvIn in, Quads quads, const bf16 *__restrict__ w,
                                                     const float *__restrict__ bias, int relu,
                                                     const bf16 *__restrict__ omask, bf16 *__restrict__ y, int Cout,
                                                     int B, int H, int W) {
  constexpr int CP = CS + 8, CH = CS / 8, ROWS = 8 * MR + 2, PATCH = ROWS * PW * CP, WSM = 9 * NB * CP;
  extern __shared__ __align__(16) bf16 conv_sm[];
  bf16 *const patches = conv_sm, *const weights = conv_sm + 2 * PATCH;
  const int tiles_w = (W + TW - 1) / TW, tiles_h = (H + 8 * MR - 1) / (8 * MR), tiles = B * tiles_h * tiles_w;
  const int Cin = in.channels(), co0 = blockIdx.y * NB, nslice = Cin / CS;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int steps = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x * nslice;
  // ldmatrix row addresses: A (pixels x channels, row-major), B (channels x couts, stored [cout][cin])
  const int am = (lane & 7) + 8 * ((lane >> 3) & 1), ak = 8 * (lane >> 4);
  const int bn = (lane & 7) + 8 * (lane >> 4), bk = 8 * ((lane >> 3) & 1);
  auto tile_at = [&](int step, int &b, int &i0, int &j0) {
    int t = blockIdx.x + step / nslice * gridDim.x;
    b = t / (tiles_h * tiles_w);
    t -= b * tiles_h * tiles_w;
    i0 = t / tiles_w * 8 * MR;
    j0 = t % tiles_w * TW;
  };
  // Channel n of a group of 32 goes to row 8 ((n mod 8) / 2) + 2 (n / 8) + n mod 2 of the staged
  // weights: a lane's columns of the four n-blocks are then eight neighbouring channels, 16 bytes
  // of a pixel.
  auto copy_weights = [&](bf16 *to, int c0) {
    for (int q = threadIdx.x; q < 9 * NB * CH; q += THREADS) {
      const int row = q / CH, ch = q - row * CH;   // row = tap * NB + n
      const int tap = row / NB, n = row - tap * NB;
      const int at = (n & ~31) + 8 * ((n & 7) >> 1) + 2 * ((n & 31) >> 3) + (n & 1);
      copy16(to + (tap * NB + at) * CP + ch * 8, w + ((size_t)tap * Cout + co0 + n) * Cin + c0 + ch * 8, true);
    }
  };
  auto copy_step = [&](int step) {
    int b, i0, j0;
    tile_at(step, b, i0, j0);
    const int c0 = step % nslice * CS;
    copy_patch<CS, THREADS, ROWS>(patches + (step & 1) * PATCH, in, c0, b, i0, j0, H, W);
    if (!RESIDENT) copy_weights(weights + (step & 1) * WSM, c0);
  };
  if (RESIDENT) copy_weights(weights, 0);
  copy_step(0);
  copy_commit();
  float acc[MR][NB / 8][4];
#pragma unroll
  for (int m = 0; m < MR; ++m)
#pragma unroll
    for (int n = 0; n < NB / 8; ++n) acc[m][n][0] = acc[m][n][1] = acc[m][n][2] = acc[m][n][3] = 0.0f;
  for (int step = 0; step < steps; ++step) {
    if (step + 1 < steps) copy_step(step + 1);
    copy_commit();
    copy_wait<1>();
    __syncthreads();
    const bf16 *const patch = patches + (step & 1) * PATCH;
    const bf16 *const wsm = RESIDENT ? weights : weights + (step & 1) * WSM;
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
      const int ky = tap / 3, kx = tap - 3 * (tap / 3);
#pragma unroll
      for (int kk = 0; kk < CS; kk += 16) {
        uint32_t a[MR][4];
#pragma unroll
        for (int m = 0; m < MR; ++m) ldsm_x4(a[m], patch + ((MR * warp + m + ky) * PW + am + kx) * CP + kk + ak);
#pragma unroll
        for (int nb2 = 0; nb2 < NB / 16; ++nb2) {
          uint32_t bb[4];
          ldsm_x4(bb, wsm + (tap * NB + nb2 * 16 + bn) * CP + kk + bk);
#pragma unroll
          for (int m = 0; m < MR; ++m) {
            mma_bf16(acc[m][2 * nb2], a[m], bb[0], bb[1]);
            mma_bf16(acc[m][2 * nb2 + 1], a[m], bb[2], bb[3]);
          }
        }
      }
    }
    __syncthreads();   // this step's buffers are free for the step after next
    if ((step + 1) % nslice != 0) continue;
    int b, i0, j0;
    tile_at(step, b, i0, j0);
    const int g = lane >> 2, tq = lane & 3;
#pragma unroll
    for (int q = 0; q < NB / 32; ++q) {
      const int co = co0 + 32 * q + 8 * tq;
      const bool own = !QUADS || co0 + 32 * q >= quads.y0, sums = QUADS && co0 + 32 * q < quads.C;
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int j = j0 + g + 8 * hh;
        uint4 out[MR];
#pragma unroll
        for (int m = 0; m < MR; ++m) {
          const int i = i0 + MR * warp + m;
          float v[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            v[u] = acc[m][4 * q + u / 2][2 * hh + (u & 1)] + (bias ? bias[co + u] : 0.0f);
            acc[m][4 * q + u / 2][2 * hh + (u & 1)] = 0.0f;   // the next tile's
            if (relu) v[u] = fmaxf(v[u], 0.0f);
          }
          out[m] = pack8(v);
          if (!own || i >= H || j >= W) continue;
          const int Cy = QUADS ? Cout - quads.y0 : Cout;
          const size_t off = (((size_t)b * H + i) * W + j) * Cy + (QUADS ? co - quads.y0 : co);
          if (omask) out[m] = relu_mask8(out[m], *reinterpret_cast<const uint4 *>(omask + off));
          *reinterpret_cast<uint4 *>(y + off) = out[m];
        }
        if constexpr (QUADS) {
          static_assert(MR == 2, "a warp has both rows of a block");
          if (!sums) continue;
          // (row, column) in the order (0, 0), (0, 1), (1, 0), (1, 1)
          float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
          for (int m = 0; m < 2; ++m) {
            const uint4 o = make_uint4(__shfl_down_sync(0xffffffffu, out[m].x, 4), __shfl_down_sync(0xffffffffu, out[m].y, 4),
                                       __shfl_down_sync(0xffffffffu, out[m].z, 4), __shfl_down_sync(0xffffffffu, out[m].w, 4));
            float f[8], r[8];
            unpack8(out[m], f);
            unpack8(o, r);
#pragma unroll
            for (int u = 0; u < 8; ++u) s[u] = s[u] + f[u] + r[u];
          }
          const int i = i0 + 2 * warp;
          if ((g & 1) || i >= H || j >= W) continue;   // H and W are even: the block is all inside
#pragma unroll
          for (int u = 0; u < 8; ++u) s[u] *= quads.scale;
          const size_t off = (((size_t)b * (H / 2) + i / 2) * (W / 2) + j / 2) * quads.C + co;
          uint4 sum = pack8(s);
          if (quads.mask) sum = relu_mask8(sum, *reinterpret_cast<const uint4 *>(quads.mask + off));
          *reinterpret_cast<uint4 *>(quads.q + off) = sum;
        }
      }
    }
  }
}

// ---- weight gradient ----
// part[cta][tap][co][ci] = sum over the CTA's pixel tiles of dy[p, co] * x[p + tap offset, ci] (dy
// masked by its ReLU where it was made).  grid = (ctas over pixel tiles, (Cout / CO) * (Cin / CI)).
// A tile's operands are copied two tiles ahead of their use.  A CTA's pixel ranges and the order
// of their sums do not depend on CO and CI, which follow from how many CTAs they leave.
//
// Bound: the chain of a CTA's tiles (its sum's order is fixed).  Waiting for each tile's loads
// took 4.3 us a tile.  Forward, backward and Adam of 16 x 128 x 128: 1.87 ms then, 1.13 ms with the
// copies ahead, of which the gradients on a stream of their own, one launch for all flipped weights and the masks
// made by their producers are a part.
constexpr int WG_STAGES = 3;
template <int CI, int CO>
constexpr int wgrad_smem() {
  return WG_STAGES * (PH * PW * (CI + 8) + TH * TW * (CO + 8)) * (int)sizeof(bf16);
}

template <int CI, int CO>
__global__ void __launch_bounds__(WG_THREADS) k_conv3x3_wgrad(ConvIn in, const bf16 *__restrict__ dy,
                                                              int Cout, int B, int H, int W, float *__restrict__ part) {
  constexpr int CP = CI + 8, DP = CO + 8, PATCH = PH * PW * CP, DYS = TH * TW * DP;
  extern __shared__ __align__(16) bf16 wg_sm[];
  const int Cin = in.channels(), nci = Cin / CI;
  const int co0 = (blockIdx.y / nci) * CO, ci0 = (blockIdx.y % nci) * CI;
  const int tiles_w = (W + TW - 1) / TW, tiles_h = (H + TH - 1) / TH, tiles = B * tiles_h * tiles_w;
  const int tap = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ky = tap / 3, kx = tap - 3 * (tap / 3);
  // A = dy^T (couts x pixels) from [pixel][cout]; B = x (pixels x cins) from [pixel][cin]
  const int apx = (lane & 7) + 8 * (lane >> 4), amo = 8 * ((lane >> 3) & 1);
  const int bpx = (lane & 7) + 8 * ((lane >> 3) & 1), bno = 8 * (lane >> 4);
  float acc[CO / 16][CI / 8][4];
#pragma unroll
  for (int m = 0; m < CO / 16; ++m)
#pragma unroll
    for (int n = 0; n < CI / 8; ++n) acc[m][n][0] = acc[m][n][1] = acc[m][n][2] = acc[m][n][3] = 0.0f;
  auto copy_tile = [&](int t, int stage) {
    bf16 *const patch = wg_sm + stage * (PATCH + DYS), *const dys = patch + PATCH;
    int r = t;
    const int b = r / (tiles_h * tiles_w);
    r -= b * tiles_h * tiles_w;
    const int i0 = (r / tiles_w) * TH, j0 = (r % tiles_w) * TW;
    copy_patch<CI, WG_THREADS, PH>(patch, in, ci0, b, i0, j0, H, W);
    for (int q = threadIdx.x; q < TH * TW * (CO / 8); q += WG_THREADS) {
      const int pix = q / (CO / 8), ch = q - pix * (CO / 8);
      const int ii = i0 + pix / TW, jj = j0 + pix % TW;
      const bool inside = ii < H && jj < W;
      copy16(dys + pix * DP + ch * 8, inside ? dy + (((size_t)b * H + ii) * W + jj) * Cout + co0 + ch * 8 : dy, inside);
    }
  };
  int next = blockIdx.x, fill = 0;
#pragma unroll
  for (int q = 0; q < WG_STAGES - 1; ++q, next += gridDim.x) {
    if (next < tiles) copy_tile(next, fill);
    copy_commit();
    ++fill;
  }
  int use = 0;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x, next += gridDim.x) {
    copy_wait<WG_STAGES - 2>();
    __syncthreads();   // this tile is there for all, and the stage filled next is free
    if (next < tiles) copy_tile(next, fill);
    copy_commit();
    if (++fill == WG_STAGES) fill = 0;
    const bf16 *const patch = wg_sm + use * (PATCH + DYS), *const dys = patch + PATCH;
    if (++use == WG_STAGES) use = 0;
#pragma unroll 4
    for (int row = 0; row < TH; ++row) {
      uint32_t a[CO / 16][4];
#pragma unroll
      for (int mb = 0; mb < CO / 16; ++mb) ldsm_x4_t(a[mb], dys + (row * TW + apx) * DP + mb * 16 + amo);
#pragma unroll
      for (int nb2 = 0; nb2 < CI / 16; ++nb2) {
        uint32_t bb[4];
        ldsm_x4_t(bb, patch + ((row + ky) * PW + bpx + kx) * CP + nb2 * 16 + bno);
#pragma unroll
        for (int mb = 0; mb < CO / 16; ++mb) {
          mma_bf16(acc[mb][2 * nb2], a[mb], bb[0], bb[1]);
          mma_bf16(acc[mb][2 * nb2 + 1], a[mb], bb[2], bb[3]);
        }
      }
    }
  }
  const int g = lane >> 2, tq = lane & 3;
  float *dst = part + ((size_t)blockIdx.x * 9 + tap) * Cout * Cin;
#pragma unroll
  for (int mb = 0; mb < CO / 16; ++mb)
#pragma unroll
    for (int nb = 0; nb < CI / 8; ++nb)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int co = co0 + mb * 16 + g + 8 * hh, ci = ci0 + nb * 8 + 2 * tq;
        *reinterpret_cast<float2 *>(dst + (size_t)co * Cin + ci) = make_float2(acc[mb][nb][2 * hh], acc[mb][nb][2 * hh + 1]);
      }
}

// out[k] = sum_{s < nparts} part[s * n + k], in order
__global__ void k_reduce_parts(const float *__restrict__ part, int nparts, int n, float *__restrict__ out) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    float s = 0.0f;
    int q = 0;
    for (; q + 16 <= nparts; q += 16) {   // sixteen loads in flight
      float v[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) v[u] = part[(size_t)(q + u) * n + k];
#pragma unroll
      for (int u = 0; u < 16; ++u) s += v[u];
    }
    for (; q < nparts; ++q) s += part[(size_t)q * n + k];
    out[k] = s;
  }
}

// The same for few outputs (n <= 128), a block per sum: it brings the parts to shared memory in
// rows of 64, then a thread adds an output's in order.  All bias gradients and the head's in one
// launch: one block each, 9 us one after the other on the weight gradients' stream.
constexpr int RS_ROWS = 64, RS_MAX = 128, FEW_SUMS = NLAYERS + 1;
struct FewSums {
  const float *part[FEW_SUMS];
  float *out[FEW_SUMS];
  int nparts[FEW_SUMS], n[FEW_SUMS];
};
__global__ void __launch_bounds__(256) k_reduce_few(FewSums f) {
  __shared__ float rows[RS_ROWS * RS_MAX];
  const float *__restrict__ const part = f.part[blockIdx.x];
  const int nparts = f.nparts[blockIdx.x], n = f.n[blockIdx.x];
  float s = 0.0f;
  for (int q0 = 0; q0 < nparts; q0 += RS_ROWS) {
    const int nq = min(RS_ROWS, nparts - q0);
    __syncthreads();
#pragma unroll 8
    for (int e = threadIdx.x; e < nq * n; e += 256) rows[e] = part[(size_t)q0 * n + e];
    __syncthreads();
    if ((int)threadIdx.x < n) {
#pragma unroll 16
      for (int q = 0; q < nq; ++q) s += rows[q * n + threadIdx.x];
    }
  }
  if ((int)threadIdx.x < n) f.out[blockIdx.x][threadIdx.x] = s;
}

// part[cta][c] = sum over the CTA's pixels of dy[p, c]
__global__ void __launch_bounds__(256) k_bias_grad(const bf16 *__restrict__ dy, int C, long long P,
                                                   float *__restrict__ part) {
  __shared__ float red[256];
  const int lanes = 256 / C;   // pixels in flight per CTA
  const int c = threadIdx.x % C, l = threadIdx.x / C;
  float s = 0.0f;
  if (l < lanes) {
    const long long stride = (long long)gridDim.x * lanes;
    long long p = (long long)blockIdx.x * lanes + l;
    for (; p + 15 * stride < P; p += 16 * stride) {   // sixteen loads in flight
      bf16 v[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) v[u] = dy[(p + u * stride) * C + c];
#pragma unroll
      for (int u = 0; u < 16; ++u) s += __bfloat162float(v[u]);
    }
    for (; p < P; p += stride) s += __bfloat162float(dy[p * C + c]);
  }
  red[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x < C) {
    float t = 0.0f;
    for (int q = 0; q < lanes; ++q) t += red[q * C + threadIdx.x];
    part[(size_t)blockIdx.x * C + threadIdx.x] = t;
  }
}

// wt[8 - tap][ci][co] = w[tap][co][ci]: the backward-data weights of layers 1 .. NLAYERS - 1
// (blockIdx.y), at their offsets in the parameter and the flipped arrays
struct FlipLayers {
  long long w[NLAYERS], wt[NLAYERS];
  int cin[NLAYERS], cout[NLAYERS];
};
__global__ void k_flip_weights(const bf16 *__restrict__ p16, FlipLayers F, bf16 *__restrict__ flip) {
  const int l = blockIdx.y + 1, Cin = F.cin[l], Cout = F.cout[l], n = 9 * Cout * Cin;
  const bf16 *__restrict__ w = p16 + F.w[l];
  bf16 *__restrict__ wt = flip + F.wt[l];
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
    const int tap = k / (Cout * Cin), r = k - tap * Cout * Cin, co = r / Cin, ci = r - co * Cin;
    wt[((size_t)(8 - tap) * Cin + ci) * Cout + co] = w[k];
  }
}

// ---- pooling, and the gradients of the concatenation's parts ----
// y[b, I, J, :] = mean of x over the 2 x 2 block; 8 channels per thread
__global__ void k_pool(const bf16 *__restrict__ x, int C, int B, int H, int W, bf16 *__restrict__ y) {
  const int h = H / 2, w = W / 2, CH = C / 8;
  const long long n = (long long)B * h * w * CH;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int ch = (int)(k % CH);
    long long p = k / CH;
    const int J = (int)(p % w);
    p /= w;
    const int I = (int)(p % h);
    const int b = (int)(p / h);
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      float f[8];
      unpack8(*reinterpret_cast<const uint4 *>(x + (((size_t)b * H + 2 * I + (d >> 1)) * W + 2 * J + (d & 1)) * C + ch * 8), f);
#pragma unroll
      for (int q = 0; q < 8; ++q) s[q] += f[q];
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) s[q] *= 0.25f;
    *reinterpret_cast<uint4 *>(y + (((size_t)b * h + I) * w + J) * C + ch * 8) = pack8(s);
  }
}

// dx[b, i, j, :] += dy[b, i/2, j/2, :] / 4, then zero where ymask <= 0 (dx's own ReLU)
__global__ void k_pool_back_add(const bf16 *__restrict__ dy, int C, int B, int H, int W,
                                const bf16 *__restrict__ ymask, bf16 *__restrict__ dx) {
  const int h = H / 2, w = W / 2, CH = C / 8;
  const long long n = (long long)B * H * W * CH;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int ch = (int)(k % CH);
    long long p = k / CH;
    const int j = (int)(p % W);
    p /= W;
    const int i = (int)(p % H);
    const int b = (int)(p / H);
    float a[8], d[8];
    bf16 *dst = dx + (((size_t)b * H + i) * W + j) * C + ch * 8;
    unpack8(*reinterpret_cast<const uint4 *>(dst), a);
    unpack8(*reinterpret_cast<const uint4 *>(dy + (((size_t)b * h + i / 2) * w + j / 2) * C + ch * 8), d);
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] += 0.25f * d[q];
    *reinterpret_cast<uint4 *>(dst) = relu_mask8(pack8(a), *reinterpret_cast<const uint4 *>(ymask + (dst - dx)));
  }
}

// du[b, I, J, :] = sum of dc[b, 2I + di, 2J + dj, 0:Cu], zero where umask <= 0 (du's ReLU);
// ds[b, i, j, :] = dc[b, i, j, Cu:]
__global__ void k_upcat_back(const bf16 *__restrict__ dc, int Cu, int Cs, int B, int H, int W,
                             const bf16 *__restrict__ umask, bf16 *__restrict__ du, bf16 *__restrict__ ds) {
  const int C = Cu + Cs, h = H / 2, w = W / 2;
  const long long nu = (long long)B * h * w * (Cu / 8), ns = (long long)B * H * W * (Cs / 8);
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < nu + ns;
       k += (long long)gridDim.x * blockDim.x) {
    if (k < nu) {
      const int CH = Cu / 8, ch = (int)(k % CH);
      long long p = k / CH;
      const int J = (int)(p % w);
      p /= w;
      const int I = (int)(p % h);
      const int b = (int)(p / h);
      float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int d = 0; d < 4; ++d) {
        float f[8];
        unpack8(*reinterpret_cast<const uint4 *>(dc + (((size_t)b * H + 2 * I + (d >> 1)) * W + 2 * J + (d & 1)) * C + ch * 8), f);
#pragma unroll
        for (int q = 0; q < 8; ++q) s[q] += f[q];
      }
      const size_t off = (((size_t)b * h + I) * w + J) * Cu + ch * 8;
      *reinterpret_cast<uint4 *>(du + off) = relu_mask8(pack8(s), *reinterpret_cast<const uint4 *>(umask + off));
    } else {
      const long long kk = k - nu;
      const int CH = Cs / 8, ch = (int)(kk % CH);
      const long long p = kk / CH;
      *reinterpret_cast<uint4 *>(ds + p * Cs + ch * 8) = *reinterpret_cast<const uint4 *>(dc + p * C + Cu + ch * 8);
    }
  }
}

// ---- input packing, head, loss ----
// x16[p, 0:8] = bf16(in[p, 0:8]), x16[p, 8:16] = 0
__global__ void k_pack_input(const float *__restrict__ in, long long P, bf16 *__restrict__ x16) {
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P; p += (long long)gridDim.x * blockDim.x) {
    float f[8];
    const float4 a = reinterpret_cast<const float4 *>(in)[2 * p], b = reinterpret_cast<const float4 *>(in)[2 * p + 1];
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w;
    f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    reinterpret_cast<uint4 *>(x16)[2 * p] = pack8(f);
    reinterpret_cast<uint4 *>(x16)[2 * p + 1] = make_uint4(0u, 0u, 0u, 0u);
  }
}

// y[p, o] = bh[o] + sum_c d1[p, c] * Wh[o, c]
__global__ void k_head(const bf16 *__restrict__ d1, const float *__restrict__ wh, long long P, float *__restrict__ y) {
  __shared__ float ws[HEAD_COUT * HEAD_CIN + HEAD_COUT];
  for (int q = threadIdx.x; q < HEAD_COUT * HEAD_CIN + HEAD_COUT; q += blockDim.x) ws[q] = wh[q];
  __syncthreads();
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P; p += (long long)gridDim.x * blockDim.x) {
    float y0 = ws[2 * HEAD_CIN], y1 = ws[2 * HEAD_CIN + 1];
#pragma unroll
    for (int ch = 0; ch < HEAD_CIN / 8; ++ch) {
      float f[8];
      unpack8(reinterpret_cast<const uint4 *>(d1 + p * HEAD_CIN)[ch], f);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        y0 = fmaf(f[q], ws[ch * 8 + q], y0);
        y1 = fmaf(f[q], ws[HEAD_CIN + ch * 8 + q], y1);
      }
    }
    reinterpret_cast<float2 *>(y)[p] = make_float2(y0, y1);
  }
}

// per CTA: {sum w (y - t)^2, sum w}
__global__ void __launch_bounds__(256) k_loss_parts(const float *__restrict__ y, const float *__restrict__ t,
                                                    const float *__restrict__ wgt, long long P, float *__restrict__ part) {
  __shared__ float r0[256], r1[256];
  float s0 = 0.0f, s1 = 0.0f;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P; p += (long long)gridDim.x * blockDim.x) {
    const float w = wgt ? wgt[p] : 1.0f;
    const float2 a = reinterpret_cast<const float2 *>(y)[p], b = reinterpret_cast<const float2 *>(t)[p];
    s0 += w * ((a.x - b.x) * (a.x - b.x) + (a.y - b.y) * (a.y - b.y));
    s1 += w;
  }
  r0[threadIdx.x] = s0;
  r1[threadIdx.x] = s1;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      r0[threadIdx.x] += r0[threadIdx.x + o];
      r1[threadIdx.x] += r1[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = r0[0];
    part[2 * blockIdx.x + 1] = r1[0];
  }
}

// sums = {ordered sum of the loss parts, sum of weights, loss = sums[0] / (2 sums[1])}
__global__ void __launch_bounds__(256) k_loss_finish(const float *__restrict__ part, int nparts,
                                                     float *__restrict__ sums) {
  __shared__ float p[2 * 256];   // nparts <= 256
  for (int q = threadIdx.x; q < 2 * nparts; q += 256) p[q] = part[q];
  __syncthreads();
  if (threadIdx.x == 0) {
    float a = 0.0f, b = 0.0f;
#pragma unroll 16
    for (int q = 0; q < nparts; ++q) {
      a += p[2 * q];
      b += p[2 * q + 1];
    }
    sums[0] = a;
    sums[1] = b;
    sums[2] = b > 0.0f ? a / (2.0f * b) : 0.0f;
  }
}

// dy = w (y - t) / sum w;  dd1[p, c] = sum_o dy[p, o] Wh[o, c], zero where d1 <= 0 (its ReLU);
// part[cta] = {dWh[2][32], dbh[2]} partial sums
__global__ void __launch_bounds__(256) k_head_back(const bf16 *__restrict__ d1, const float *__restrict__ y,
                                                   const float *__restrict__ t, const float *__restrict__ wgt,
                                                   const float *__restrict__ sums, const float *__restrict__ wh,
                                                   long long P, bf16 *__restrict__ dd1, float *__restrict__ part) {
  constexpr int NG = HEAD_COUT * HEAD_CIN + HEAD_COUT;
  __shared__ float red[NG][33];
  float g[NG];
#pragma unroll
  for (int q = 0; q < NG; ++q) g[q] = 0.0f;
  const float inv = sums[1] > 0.0f ? 1.0f / sums[1] : 0.0f;
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < P; p += (long long)gridDim.x * blockDim.x) {
    const float w = (wgt ? wgt[p] : 1.0f) * inv;
    const float2 a = reinterpret_cast<const float2 *>(y)[p], b = reinterpret_cast<const float2 *>(t)[p];
    const float e0 = w * (a.x - b.x), e1 = w * (a.y - b.y);
#pragma unroll
    for (int ch = 0; ch < HEAD_CIN / 8; ++ch) {
      float f[8], o[8];
      unpack8(reinterpret_cast<const uint4 *>(d1 + p * HEAD_CIN)[ch], f);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int c = ch * 8 + q;
        o[q] = e0 * wh[c] + e1 * wh[HEAD_CIN + c];
        g[c] = fmaf(e0, f[q], g[c]);
        g[HEAD_CIN + c] = fmaf(e1, f[q], g[HEAD_CIN + c]);
      }
      reinterpret_cast<uint4 *>(dd1 + p * HEAD_CIN)[ch] =
          relu_mask8(pack8(o), reinterpret_cast<const uint4 *>(d1 + p * HEAD_CIN)[ch]);
    }
    g[2 * HEAD_CIN] += e0;
    g[2 * HEAD_CIN + 1] += e1;
  }
  // warp sums, then the 8 warps in order
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NG; ++q) {
    float v = g[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[q][warp] = v;
  }
  __syncthreads();
  if (threadIdx.x < NG) {
    float s = 0.0f;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) s += red[threadIdx.x][q];
    part[(size_t)blockIdx.x * NG + threadIdx.x] = s;
  }
}

// Adam with bias correction; the BF16 copy of every parameter follows the FP32 master
__global__ void k_adam(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m, float *__restrict__ v,
                       long long n, float lr, float b1, float b2, float eps, float c1, float c2,
                       bf16 *__restrict__ p16) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const float gk = g[k];
    const float mk = b1 * m[k] + (1.0f - b1) * gk;
    const float vk = b2 * v[k] + (1.0f - b2) * gk * gk;
    m[k] = mk;
    v[k] = vk;
    const float pk = p[k] - lr * (mk / c1) / (sqrtf(vk / c2) + eps);
    p[k] = pk;
    p16[k] = __float2bfloat16_rn(pk);
  }
}

__global__ void k_to_bf16(const float *__restrict__ p, long long n, bf16 *__restrict__ p16) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
    p16[k] = __float2bfloat16_rn(p[k]);
}

// ---- the SSA side: features and the velocity from the network output ----
__global__ void k_features(int Mx, int My, int stride, const double *__restrict__ H, const double *__restrict__ bed,
                           const double *__restrict__ tauc, const double2 *__restrict__ hardness,
                           const int8_t *__restrict__ mask, const double2 *__restrict__ taud,
                           float *__restrict__ out, int height, int width) {
  const long long n = (long long)height * width;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    const int I = (int)(q / width), J = (int)(q % width);
    const int i = I * stride, j = J * stride;
    float f[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (i < Mx && j < My) {
      const size_t k = (size_t)i * My + j;
      const int m = mask[k];
      const double2 hb = hardness[k];
      const double hv = fmax(hb.x, hb.y);
      f[0] = (float)(H[k] * 1e-3);
      f[1] = (float)(bed[k] * 1e-3);
      f[2] = (float)log(fmax(tauc[k], 1.0) / 5.0e4);
      f[3] = (m == 2 || m == 3) && hv > 0.0 ? (float)(hv * 1e-8) : 0.0f;
      f[4] = m == 2 ? 1.0f : 0.0f;
      f[5] = m == 3 ? 1.0f : 0.0f;
      f[6] = (float)(taud[k].x * 1e-5);
      f[7] = (float)(taud[k].y * 1e-5);
    }
    float4 *o = reinterpret_cast<float4 *>(out + q * 8);
    o[0] = make_float4(f[0], f[1], f[2], f[3]);
    o[1] = make_float4(f[4], f[5], f[6], f[7]);
  }
}

// vel(i, j) = 10 m/yr * sinh(y) at the coarse points, bilinear in between (stride 1 or 2)
__global__ void k_velocity(const float *__restrict__ y, int height, int width, int stride, int Mx, int My,
                           double secpera, double2 *__restrict__ vel) {
  const long long n = (long long)Mx * My;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(k / My), j = (int)(k % My);
    const int I0 = i / stride, J0 = j / stride;
    const int I1 = min(I0 + (i % stride ? 1 : 0), height - 1), J1 = min(J0 + (j % stride ? 1 : 0), width - 1);
    double u = 0.0, v = 0.0;
    const int Is[2] = {I0, I1}, Js[2] = {J0, J1};
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const float2 o = reinterpret_cast<const float2 *>(y)[(size_t)Is[a] * width + Js[b]];
        u += 10.0 * sinh((double)o.x);
        v += 10.0 * sinh((double)o.y);
      }
    vel[k] = make_double2(0.25 * u / secpera, 0.25 * v / secpera);
  }
}

// ---- the learned preconditioner correction: the residual's image and the correction ----
constexpr int PC_THREADS = 256;

// channels 6, 7 of the image = the stride x stride block means of s = D^-1 r (the
// block-Jacobi-scaled residual, in velocity units); per block the partial sum of their squares
__global__ void __launch_bounds__(PC_THREADS) k_pc_image(int Mx, int My, int stride, const double2 *__restrict__ r,
                                                          const double4 *__restrict__ dinv, float *__restrict__ img,
                                                          int height, int width, double *__restrict__ part,
                                                          const int *done) {
  if (done && *done) return;
  double acc = 0.0;
  const long long n = (long long)height * width;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    const int I = (int)(q / width), J = (int)(q % width);
    double su = 0.0, sv = 0.0;
    int cnt = 0;
    for (int a = 0; a < stride; ++a)
      for (int b = 0; b < stride; ++b) {
        const int i = I * stride + a, j = J * stride + b;
        if (i < Mx && j < My) {
          const size_t k = (size_t)i * My + j;
          const double4 d = dinv[k];
          const double2 rk = r[k];
          su += d.x * rk.x + d.y * rk.y;
          sv += d.z * rk.x + d.w * rk.y;
          ++cnt;
        }
      }
    if (cnt > 0) {
      su /= cnt;
      sv /= cnt;
    }
    img[q * 8 + 6] = (float)su;
    img[q * 8 + 7] = (float)sv;
    acc += su * su + sv * sv;
  }
  __shared__ double sh[PC_THREADS / 32];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < PC_THREADS / 32; ++w) t += sh[w];
    part[blockIdx.x] = t;
  }
}

// rho = RMS of the residual channels (every block sums the partials in the same order);
// channels 6, 7 scaled by 1 / rho; block 0 stores rho
__global__ void __launch_bounds__(PC_THREADS) k_pc_scale(float *__restrict__ img, int height, int width,
                                                          const double *__restrict__ part, int nparts,
                                                          double *__restrict__ rho_out, const int *done) {
  if (done && *done) return;
  __shared__ double rho_sh;
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int b = 0; b < nparts; ++b) t += part[b];
    rho_sh = sqrt(t / (2.0 * (double)height * width));
    if (blockIdx.x == 0) *rho_out = rho_sh;
  }
  __syncthreads();
  const double rho = rho_sh;
  const float inv = rho > 0.0 ? (float)(1.0 / rho) : 0.0f;
  const long long n = (long long)height * width;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    img[q * 8 + 6] *= inv;
    img[q * 8 + 7] *= inv;
  }
}

// d = rho * (the network's output interpolated to the grid, as k_velocity interpolates)
__global__ void k_pc_expand(const float *__restrict__ y, int height, int width, int stride, int Mx, int My,
                            const double *__restrict__ rho, double2 *__restrict__ d, const int *done) {
  if (done && *done) return;
  const double s = *rho;
  const long long n = (long long)Mx * My;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(k / My), j = (int)(k % My);
    const int I0 = i / stride, J0 = j / stride;
    const int I1 = min(I0 + (i % stride ? 1 : 0), height - 1), J1 = min(J0 + (j % stride ? 1 : 0), width - 1);
    double u = 0.0, v = 0.0;
    const int Is[2] = {I0, I1}, Js[2] = {J0, J1};
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        const float2 o = reinterpret_cast<const float2 *>(y)[(size_t)Is[a] * width + Js[b]];
        u += (double)o.x;
        v += (double)o.y;
      }
    d[k] = make_double2(0.25 * s * u, 0.25 * s * v);
  }
}

}  // namespace pism_unet

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
using namespace pism_unet;

struct pism_gpu_unet {
  int device = 0;
  int maxB = 0, maxH = 0, maxW = 0;
  cudaStream_t stream = nullptr;
  long long nparam = 0;
  std::vector<long long> w_off, b_off, flip_off;   // offsets into the parameter / flipped arrays
  long long head_off = 0;
  float *p32 = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;
  bf16 *p16 = nullptr, *flip = nullptr;
  long long flip_n = 0;
  float *wg_part = nullptr;   // weight-gradient partial sums
  size_t wg_part_n = 0;
  float *small_part = nullptr;   // head / loss partial sums
  float *bias_part = nullptr;    // bias partial sums, BIAS_MAX_CTAS x RS_MAX a layer
  FewSums few = {};              // the sums of a backward's last launch
  cudaStream_t side = nullptr;   // the weight gradients, beside the data gradients
  cudaEvent_t ready[NLAYERS] = {}, side_done = nullptr;
  float *sums = nullptr;
  float *sums_host = nullptr;
  // activations (bf16) and their gradients
  bf16 *in16 = nullptr;
  bf16 *act[NLAYERS] = {};
  bf16 *p1 = nullptr, *p2 = nullptr, *p3 = nullptr;
  float *y = nullptr;
  bf16 *dd1 = nullptr, *dc1 = nullptr, *dd2 = nullptr, *de1 = nullptr, *dc2 = nullptr, *dd3 = nullptr,
       *de2 = nullptr, *dc3 = nullptr, *dbt = nullptr, *de3 = nullptr, *dp3 = nullptr, *de3a = nullptr,
       *dp2 = nullptr, *de2a = nullptr, *dp1 = nullptr, *de1a = nullptr;
  int B = 0, H = 0, W = 0;   // shape of the last forward
  bool have_forward = false, have_grad = false;
  long long adam_t = 0;
  std::string err;
};

namespace {

int ufail(pism_gpu_unet *h, int code, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  if (h) h->err = buf;
  return code;
}

#define UCK(h, call)                                                                                  \
  do {                                                                                                \
    cudaError_t e_ = (call);                                                                          \
    if (e_ != cudaSuccess) return ufail(h, PISM_GPU_SSA_ECUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
  } while (0)

struct UDevice {
  int prev = -1;
  explicit UDevice(int dev) {
    cudaGetDevice(&prev);
    if (prev != dev) cudaSetDevice(dev);
  }
  ~UDevice() {
    int cur = -1;
    cudaGetDevice(&cur);
    if (prev >= 0 && cur != prev) cudaSetDevice(prev);
  }
};

int grid_for(long long n, int threads = 256) {
  return (int)std::max(1LL, std::min((n + threads - 1) / threads, 148LL * 16));
}

template <class T>
cudaError_t ualloc(T **p, size_t count) {
  return cudaMalloc((void **)p, std::max<size_t>(count, 1) * sizeof(T));
}

// level-l pixel count of a B x H x W image
inline long long pixels(int B, int H, int W, int l) { return (long long)B * (H >> l) * (W >> l); }

constexpr int UNET_SMS = 148;

// one kernel form: its dynamic shared memory (granted when a handle is created) and its launch
template <int CS, int NB, int MR, bool RESIDENT, bool QUADS = false>
struct Conv {
  static constexpr int smem = conv_smem<CS, NB, MR, RESIDENT>();
  static bool allow() {
    return cudaFuncSetAttribute((const void *)k_conv3x3<CS, NB, MR, RESIDENT, QUADS>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess;
  }
  static void launch(cudaStream_t s, const ConvIn &in, const Quads &quads, const bf16 *w, const float *bias, int relu, const bf16 *omask,
                     bf16 *y, int Cout, int B, int H, int W) {
    const int tiles = B * ((H + 8 * MR - 1) / (8 * MR)) * ((W + TW - 1) / TW), ny = Cout / NB;
    // Where the weights stay, as many CTAs as are resident at once, each with the same number of
    // tiles (a first tile cannot overlap its loads).  Several slices pipeline within a tile and
    // fetch their weights for each: a tile a CTA, whose start and end then overlap its
    // neighbours' (forward of 1 x 408 x 408: 269 us; equal shares 289, pairs of tiles 310).
    const int most = std::max(1, UNET_SMS * std::min(3, (220 * 1024) / smem) / ny);
    const int per = RESIDENT ? (tiles + most - 1) / most : 1, ctas = (tiles + per - 1) / per;
    k_conv3x3<CS, NB, MR, RESIDENT, QUADS><<<dim3(ctas, ny), THREADS, smem, s>>>(in, quads, w, bias, relu, omask, y, Cout,
                                                                                 B, H, W);
  }
};
template <int CI, int CO>
struct Wgrad {
  static constexpr int smem = wgrad_smem<CI, CO>();
  static bool allow() {
    return cudaFuncSetAttribute((const void *)k_conv3x3_wgrad<CI, CO>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                smem) == cudaSuccess;
  }
  static void launch(cudaStream_t s, const ConvIn &in, const bf16 *dy, int Cout, int B, int H, int W, int ctas,
                     float *part) {
    k_conv3x3_wgrad<CI, CO><<<dim3(ctas, (Cout / CO) * (in.channels() / CI)), WG_THREADS, smem, s>>>(in, dy, Cout, B, H,
                                                                                                    W, part);
  }
};
bool allow_kernels() {
  return Conv<32, 32, 2, true>::allow() && Conv<32, 32, 2, false>::allow() && Conv<32, 32, 1, true>::allow() &&
         Conv<32, 32, 2, true, true>::allow() && Conv<32, 32, 2, false, true>::allow() && Conv<32, 32, 1, false>::allow() && Conv<16, 32, 2, true>::allow() && Conv<16, 32, 1, true>::allow() &&
         Wgrad<32, 32>::allow() && Wgrad<32, 16>::allow() && Wgrad<16, 16>::allow();
}

// whether a layer's tiles are 16 x 16 pixels: where that leaves every SM a CTA; else 8 x 16
bool tall_tiles(int Cout, int B, int H, int W) {
  return (long long)B * ((H + 15) / 16) * ((W + TW - 1) / TW) * (Cout / 32) >= UNET_SMS;
}

// the weights stay in shared memory where the layer is one slice
void conv(cudaStream_t s, const ConvIn &in, const bf16 *w, const float *bias, int relu, const bf16 *omask,
          bf16 *y, int Cout, int B, int H, int W) {
  const int Cin = in.channels();
  const bool tall = tall_tiles(Cout, B, H, W);
  const Quads none{};
  if (Cin == 16) {
    if (tall) Conv<16, 32, 2, true>::launch(s, in, none, w, bias, relu, omask, y, Cout, B, H, W);
    else Conv<16, 32, 1, true>::launch(s, in, none, w, bias, relu, omask, y, Cout, B, H, W);
  } else if (Cin == 32) {
    if (tall) Conv<32, 32, 2, true>::launch(s, in, none, w, bias, relu, omask, y, Cout, B, H, W);
    else Conv<32, 32, 1, true>::launch(s, in, none, w, bias, relu, omask, y, Cout, B, H, W);
  } else {
    if (tall) Conv<32, 32, 2, false>::launch(s, in, none, w, bias, relu, omask, y, Cout, B, H, W);
    else Conv<32, 32, 1, false>::launch(s, in, none, w, bias, relu, omask, y, Cout, B, H, W);
  }
}

// a layer of 32 channels or more with tall tiles, and the 2 x 2 sums behind it
void conv_quads(cudaStream_t s, const ConvIn &in, const Quads &quads, const bf16 *w, const float *bias, int relu, bf16 *y,
                int Cout, int B, int H, int W) {
  if (in.channels() == 32) Conv<32, 32, 2, true, true>::launch(s, in, quads, w, bias, relu, nullptr, y, Cout, B, H, W);
  else Conv<32, 32, 2, false, true>::launch(s, in, quads, w, bias, relu, nullptr, y, Cout, B, H, W);
}

// dW: the channel blocks are halved while that still leaves SMs without a CTA
void conv_wgrad(pism_gpu_unet *h, cudaStream_t s, const ConvIn &in, const bf16 *dy, int Cout, int B, int H, int W,
                float *dW) {
  const int Cin = in.channels();
  const int tiles = B * ((H + TH - 1) / TH) * ((W + TW - 1) / TW);
  const int ctas = std::min(tiles, WG_MAX_CTAS);
  const int blocks = ctas * (Cout / 32) * std::max(1, Cin / 32);   // with blocks of 32 x 32
  const bool half = blocks < 2 * UNET_SMS, quarter = blocks < UNET_SMS;
  if (Cin % 32 != 0 || quarter) {   // 16 input channels: the first layer only, one block of 32 x 32
    Wgrad<16, 16>::launch(s, in, dy, Cout, B, H, W, ctas, h->wg_part);
  } else if (half) {
    Wgrad<32, 16>::launch(s, in, dy, Cout, B, H, W, ctas, h->wg_part);
  } else {
    Wgrad<32, 32>::launch(s, in, dy, Cout, B, H, W, ctas, h->wg_part);
  }
  const int n = 9 * Cout * Cin;
  k_reduce_parts<<<grid_for(n), 256, 0, s>>>(h->wg_part, ctas, n, dW);
}

// what layer l reads: an activation, pooled where a level begins, or the decoder's concatenation of
// the level below and the skip
ConvIn input_of(const pism_gpu_unet *h, int l) {
  switch (l) {
    case 0: return {h->in16, nullptr, LAYERS[0].cin, 0};
    case 2: return {h->p1, nullptr, LAYERS[2].cin, 0};
    case 4: return {h->p2, nullptr, LAYERS[4].cin, 0};
    case 6: return {h->p3, nullptr, LAYERS[6].cin, 0};
    case 7: return {h->act[5], h->act[6], LAYERS[5].cout, LAYERS[6].cout};
    case 8: return {h->act[3], h->act[7], LAYERS[3].cout, LAYERS[7].cout};
    case 9: return {h->act[1], h->act[8], LAYERS[1].cout, LAYERS[8].cout};
    default: return {h->act[l - 1], nullptr, LAYERS[l].cin, 0};
  }
}

// layer l's partial bias gradients; the sums follow in one launch for all layers
void bias_grad(pism_gpu_unet *h, int l, const bf16 *dy, long long P) {
  const int C = LAYERS[l].cout;
  FewSums &f = h->few;
  f.nparts[l] = (int)std::min<long long>(BIAS_MAX_CTAS, std::max(1LL, P / 64));
  f.n[l] = C;
  f.out[l] = h->grad + h->b_off[l];
  float *const part = h->bias_part + (size_t)l * BIAS_MAX_CTAS * RS_MAX;
  f.part[l] = part;
  k_bias_grad<<<f.nparts[l], 256, 0, h->stream>>>(dy, C, P, part);
}

cudaError_t layer_back(pism_gpu_unet *h, int l, const bf16 *dY, bf16 *dX, const bf16 *xmask, int B, int H, int W,
                       const Quads *split);

// Layer l backward where its input is a concatenation: the gradients of the upsampled part (du, masked
// by its layer's ReLU) and of the skip (ds); dc takes the concatenation's where the tiles are not tall
cudaError_t concat_back(pism_gpu_unet *h, int l, const bf16 *dY, bf16 *du, bf16 *ds, bf16 *dc, int B, int H, int W) {
  const ConvIn in = input_of(h, l);
  if (tall_tiles(in.channels(), B, H, W)) {
    const Quads split{du, in.up, in.Cu, in.Cu, 1.0f};
    return layer_back(h, l, dY, ds, nullptr, B, H, W, &split);
  }
  const cudaError_t e = layer_back(h, l, dY, dc, nullptr, B, H, W, nullptr);
  if (e != cudaSuccess) return e;
  k_upcat_back<<<grid_for((long long)B * H * W * in.channels() / 8), 256, 0, h->stream>>>(dc, in.Cu, in.C, B, H, W, in.up, du,
                                                                                     ds);
  return cudaSuccess;
}

// the second stream and its events, from the first backward on: a network that only predicts has none
bool side_stream(pism_gpu_unet *h) {
  if (h->side_done) return true;
  bool ok = h->side || cudaStreamCreateWithFlags(&h->side, cudaStreamNonBlocking) == cudaSuccess;
  for (cudaEvent_t &e : h->ready)
    ok = ok && (e || cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess);
  return ok && cudaEventCreateWithFlags(&h->side_done, cudaEventDisableTiming) == cudaSuccess;
}

// Layer l backward: dY given, masked by the layer's ReLU; dX (masked by xmask, its own
// layer's output, where given) and db on the handle's stream, dW beside them on the second one: the
// data gradients are the only chain, and with db behind them the streams are about as long
// (with split, dX is the gradient of the skip and the other part's is made beside it; 16 x 128 x 128, kernel time: 450 and 410 us; 360 and 590 with all that is not a chain on the second).
cudaError_t layer_back(pism_gpu_unet *h, int l, const bf16 *dY, bf16 *dX, const bf16 *xmask, int B, int H, int W,
                       const Quads *split) {
  const LayerDef &L = LAYERS[l];
  cudaError_t e = cudaEventRecord(h->ready[l], h->stream);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(h->side, h->ready[l], 0);
  if (e != cudaSuccess) return e;
  if (dX && split)
    conv_quads(h->stream, {dY, nullptr, L.cout, 0}, *split, h->flip + h->flip_off[l], nullptr, 0, dX, L.cin, B, H, W);
  else if (dX) conv(h->stream, {dY, nullptr, L.cout, 0}, h->flip + h->flip_off[l], nullptr, 0, xmask, dX, L.cin, B, H, W);
  conv_wgrad(h, h->side, input_of(h, l), dY, L.cout, B, H, W, h->grad + h->w_off[l]);
  bias_grad(h, l, dY, (long long)B * H * W);
  return cudaSuccess;
}

int check_shape(pism_gpu_unet *h, int B, int H, int W) {
  if (B < 1 || H < 8 || W < 8 || H % 8 || W % 8)
    return ufail(h, PISM_GPU_SSA_EINVAL, "image %d x %d x %d: batch >= 1, height and width multiples of 8", B, H, W);
  if ((long long)B * H * W > (long long)h->maxB * h->maxH * h->maxW)
    return ufail(h, PISM_GPU_SSA_ETOOLARGE, "image %d x %d x %d exceeds the allocation (%d x %d x %d)", B, H, W,
                 h->maxB, h->maxH, h->maxW);
  return PISM_GPU_SSA_OK;
}

}  // namespace

namespace pism_unet {

void launch_features(cudaStream_t s, int Mx, int My, int stride, const double *H, const double *bed,
                     const double *tauc, const double2 *hardness, const int8_t *mask, const double2 *taud, float *out,
                     int height, int width) {
  k_features<<<grid_for((long long)height * width), 256, 0, s>>>(Mx, My, stride, H, bed, tauc, hardness, mask, taud,
                                                                  out, height, width);
}

int pc_parts(int height, int width) { return std::min(grid_for((long long)height * width, PC_THREADS), 592); }

void launch_pc_input(cudaStream_t s, int Mx, int My, int stride, const double2 *r, const double4 *dinv, float *img,
                     int height, int width, double *part, double *rho, const int *done) {
  const int nb = pc_parts(height, width);
  k_pc_image<<<nb, PC_THREADS, 0, s>>>(Mx, My, stride, r, dinv, img, height, width, part, done);
  k_pc_scale<<<nb, PC_THREADS, 0, s>>>(img, height, width, part, nb, rho, done);
}

void launch_pc_expand(cudaStream_t s, const float *y, int height, int width, int stride, int Mx, int My,
                      const double *rho, double2 *d, const int *done) {
  k_pc_expand<<<grid_for((long long)Mx * My), 256, 0, s>>>(y, height, width, stride, Mx, My, rho, d, done);
}

void launch_velocity(cudaStream_t s, const float *y, int height, int width, int stride, int Mx, int My,
                     double secpera, double2 *vel) {
  k_velocity<<<grid_for((long long)Mx * My), 256, 0, s>>>(y, height, width, stride, Mx, My, secpera, vel);
}

cudaStream_t stream_of(const pism_gpu_unet *h) { return h->stream; }
int device_of(const pism_gpu_unet *h) { return h->device; }

}  // namespace pism_unet

extern "C" {

long long pism_gpu_unet_param_count(void) { return param_count(); }

int pism_gpu_unet_create(int device, int max_batch, int max_h, int max_w, pism_gpu_unet **out) {
  if (!out || max_batch < 1 || max_h < 8 || max_w < 8 || max_h % 8 || max_w % 8) return PISM_GPU_SSA_EINVAL;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) return PISM_GPU_SSA_ECUDA;
  UDevice dg(device);
  pism_gpu_unet *h = new pism_gpu_unet();
  h->device = device;
  h->maxB = max_batch;
  h->maxH = max_h;
  h->maxW = max_w;
  h->nparam = param_count();
  long long off = 0, foff = 0;
  for (const LayerDef &L : LAYERS) {
    h->w_off.push_back(off);
    h->flip_off.push_back(foff);
    off += 9LL * L.cout * L.cin;
    foff += 9LL * L.cout * L.cin;
    h->b_off.push_back(off);
    off += L.cout;
  }
  h->head_off = off;
  h->flip_n = foff;
  size_t wg = 0;
  for (const LayerDef &L : LAYERS) wg = std::max(wg, (size_t)9 * L.cout * L.cin);
  h->wg_part_n = wg * WG_MAX_CTAS;
  const long long P0 = (long long)max_batch * max_h * max_w;
  auto P = [&](int l) { return (size_t)(P0 >> (2 * l)); };
  int rc = PISM_GPU_SSA_OK;
  auto A = [&](bf16 **p, size_t n) {
    if (rc == PISM_GPU_SSA_OK && ualloc(p, n) != cudaSuccess) rc = PISM_GPU_SSA_ENOMEM;
  };
  auto AF = [&](float **p, size_t n) {
    if (rc == PISM_GPU_SSA_OK && ualloc(p, n) != cudaSuccess) rc = PISM_GPU_SSA_ENOMEM;
  };
  AF(&h->p32, h->nparam);
  AF(&h->grad, h->nparam);
  AF(&h->m, h->nparam);
  AF(&h->v, h->nparam);
  A(&h->p16, h->nparam);
  A(&h->flip, h->flip_n);
  AF(&h->wg_part, h->wg_part_n);
  AF(&h->small_part, 256 * 130);
  AF(&h->bias_part, (size_t)NLAYERS * BIAS_MAX_CTAS * RS_MAX);
  AF(&h->sums, 4);
  if (rc == PISM_GPU_SSA_OK && cudaMallocHost((void **)&h->sums_host, 4 * sizeof(float)) != cudaSuccess)
    rc = PISM_GPU_SSA_ENOMEM;
  A(&h->in16, P(0) * 16);
  for (int l = 0; l < NLAYERS; ++l) A(&h->act[l], P(LAYERS[l].level) * LAYERS[l].cout);
  A(&h->p1, P(1) * 32);
  A(&h->p2, P(2) * 64);
  A(&h->p3, P(3) * 96);
  AF(&h->y, P(0) * 2);
  A(&h->dd1, P(0) * 32);
  A(&h->dc1, P(0) * 96);
  A(&h->dd2, P(1) * 64);
  A(&h->de1, P(0) * 32);
  A(&h->dc2, P(1) * 160);
  A(&h->dd3, P(2) * 96);
  A(&h->de2, P(1) * 64);
  A(&h->dc3, P(2) * 224);
  A(&h->dbt, P(3) * 128);
  A(&h->de3, P(2) * 96);
  A(&h->dp3, P(3) * 96);
  A(&h->de3a, P(2) * 96);
  A(&h->dp2, P(2) * 64);
  A(&h->de2a, P(1) * 64);
  A(&h->dp1, P(1) * 32);
  A(&h->de1a, P(0) * 32);
  if (rc == PISM_GPU_SSA_OK && !allow_kernels()) rc = PISM_GPU_SSA_ECUDA;
  if (rc != PISM_GPU_SSA_OK) {
    pism_gpu_unet_destroy(h);
    return rc;
  }
  cudaMemset(h->p32, 0, h->nparam * sizeof(float));
  cudaMemset(h->p16, 0, h->nparam * sizeof(bf16));
  cudaMemset(h->flip, 0, h->flip_n * sizeof(bf16));
  cudaMemset(h->m, 0, h->nparam * sizeof(float));
  cudaMemset(h->v, 0, h->nparam * sizeof(float));
  if (cudaDeviceSynchronize() != cudaSuccess) {
    pism_gpu_unet_destroy(h);
    return PISM_GPU_SSA_ECUDA;
  }
  *out = h;
  return PISM_GPU_SSA_OK;
}

int pism_gpu_unet_destroy(pism_gpu_unet *h) {
  if (!h) return PISM_GPU_SSA_OK;
  UDevice dg(h->device);
  cudaStreamSynchronize(h->stream);
  if (h->side) cudaStreamSynchronize(h->side);
  if (h->side) cudaStreamDestroy(h->side);
  if (h->side_done) cudaEventDestroy(h->side_done);
  for (cudaEvent_t e : h->ready)
    if (e) cudaEventDestroy(e);
  for (float *p : {h->p32, h->grad, h->m, h->v, h->wg_part, h->small_part, h->bias_part, h->sums, h->y}) cudaFree(p);
  for (bf16 *p : {h->p16, h->flip, h->in16, h->p1, h->p2, h->p3, h->dd1, h->dc1, h->dd2, h->de1,
                  h->dc2, h->dd3, h->de2, h->dc3, h->dbt, h->de3, h->dp3, h->de3a, h->dp2, h->de2a, h->dp1, h->de1a})
    cudaFree(p);
  for (bf16 *p : h->act) cudaFree(p);
  if (h->sums_host) cudaFreeHost(h->sums_host);
  delete h;
  return PISM_GPU_SSA_OK;
}

const char *pism_gpu_unet_last_error(const pism_gpu_unet *h) { return h ? h->err.c_str() : "null handle"; }

int pism_gpu_unet_set_stream(pism_gpu_unet *h, void *stream) {
  if (!h) return PISM_GPU_SSA_EINVAL;
  h->stream = (cudaStream_t)stream;
  return PISM_GPU_SSA_OK;
}

int pism_gpu_unet_set_params(pism_gpu_unet *h, const float *params, int where) {
  if (!h || !params) return PISM_GPU_SSA_EINVAL;
  UDevice dg(h->device);
  UCK(h, cudaMemcpyAsync(h->p32, params, h->nparam * sizeof(float),
                         where == PISM_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice, h->stream));
  k_to_bf16<<<grid_for(h->nparam), 256, 0, h->stream>>>(h->p32, h->nparam, h->p16);
  UCK(h, cudaMemsetAsync(h->m, 0, h->nparam * sizeof(float), h->stream));
  UCK(h, cudaMemsetAsync(h->v, 0, h->nparam * sizeof(float), h->stream));
  h->adam_t = 0;
  UCK(h, cudaGetLastError());
  UCK(h, cudaStreamSynchronize(h->stream));
  return PISM_GPU_SSA_OK;
}

int pism_gpu_unet_get_params(pism_gpu_unet *h, float *params, int where) {
  if (!h || !params) return PISM_GPU_SSA_EINVAL;
  UDevice dg(h->device);
  UCK(h, cudaMemcpyAsync(params, h->p32, h->nparam * sizeof(float),
                         where == PISM_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, h->stream));
  UCK(h, cudaStreamSynchronize(h->stream));
  return PISM_GPU_SSA_OK;
}

int pism_gpu_unet_forward(pism_gpu_unet *h, const float *input, int B, int H, int W, float *output) {
  if (!h || !input || !output) return PISM_GPU_SSA_EINVAL;
  int rc = check_shape(h, B, H, W);
  if (rc != PISM_GPU_SSA_OK) return rc;
  UDevice dg(h->device);
  const long long P0 = (long long)B * H * W;
  const bf16 *w = h->p16;
  const float *p = h->p32;
  auto L = [&](int l) {
    const int lev = LAYERS[l].level;
    conv(h->stream, input_of(h, l), w + h->w_off[l], p + h->b_off[l], 1, nullptr, h->act[l], LAYERS[l].cout, B, H >> lev,
         W >> lev);
  };
  // a level's last layer before the next one, and its 2 x 2 means
  auto L_pooled = [&](int l, bf16 *pooled) {
    const int lev = LAYERS[l].level, C = LAYERS[l].cout, Hl = H >> lev, Wl = W >> lev;
    if (tall_tiles(C, B, Hl, Wl)) {
      conv_quads(h->stream, input_of(h, l), {pooled, nullptr, C, 0, 0.25f}, w + h->w_off[l], p + h->b_off[l], 1, h->act[l], C,
                 B, Hl, Wl);
      return;
    }
    L(l);
    k_pool<<<grid_for(pixels(B, H, W, lev + 1) * (C / 8)), 256, 0, h->stream>>>(h->act[l], C, B, Hl, Wl, pooled);
  };
  k_pack_input<<<grid_for(P0), 256, 0, h->stream>>>(input, P0, h->in16);
  L(0);
  L_pooled(1, h->p1);
  L(2);
  L_pooled(3, h->p2);
  L(4);
  L_pooled(5, h->p3);
  for (int l = 6; l < NLAYERS; ++l) L(l);
  k_head<<<grid_for(P0), 256, 0, h->stream>>>(h->act[9], p + h->head_off, P0, h->y);
  UCK(h, cudaGetLastError());
  if (output != h->y)
    UCK(h, cudaMemcpyAsync(output, h->y, P0 * 2 * sizeof(float), cudaMemcpyDeviceToDevice, h->stream));
  h->B = B;
  h->H = H;
  h->W = W;
  h->have_forward = true;
  return PISM_GPU_SSA_OK;
}

int pism_gpu_unet_backward(pism_gpu_unet *h, const float *target, const float *weight, float *loss_host,
                           float *grad_out) {
  if (!h || !target) return PISM_GPU_SSA_EINVAL;
  if (!h->have_forward) return ufail(h, PISM_GPU_SSA_ESTATE, "backward needs a forward first");
  UDevice dg(h->device);
  if (!side_stream(h)) return ufail(h, PISM_GPU_SSA_ECUDA, "no stream for the weight gradients");
  const int B = h->B, H = h->H, W = h->W;
  const long long P0 = (long long)B * H * W;
  // weights of the backward-data convolutions
  FlipLayers fl{};
  for (int l = 1; l < NLAYERS; ++l) {
    fl.w[l] = h->w_off[l];
    fl.wt[l] = h->flip_off[l];
    fl.cin[l] = LAYERS[l].cin;
    fl.cout[l] = LAYERS[l].cout;
  }
  k_flip_weights<<<dim3(128, NLAYERS - 1), 256, 0, h->stream>>>(h->p16, fl, h->flip);
  // loss and the head
  const int lctas = (int)std::min<long long>(256, std::max(1LL, P0 / 256));
  k_loss_parts<<<lctas, 256, 0, h->stream>>>(h->y, target, weight, P0, h->small_part);
  k_loss_finish<<<1, 256, 0, h->stream>>>(h->small_part, lctas, h->sums);
  const int hctas = (int)std::min<long long>(256, std::max(1LL, P0 / 256));
  constexpr int NG = HEAD_COUT * HEAD_CIN + HEAD_COUT;
  k_head_back<<<hctas, 256, 0, h->stream>>>(h->act[9], h->y, target, weight, h->sums, h->p32 + h->head_off, P0, h->dd1,
                                            h->small_part);
  h->few.part[NLAYERS] = h->small_part;
  h->few.nparts[NLAYERS] = hctas;
  h->few.n[NLAYERS] = NG;
  h->few.out[NLAYERS] = h->grad + h->head_off;
  // decoder (every gradient masked by its layer's ReLU where it is made)
  UCK(h, concat_back(h, 9, h->dd1, h->dd2, h->de1, h->dc1, B, H, W));
  UCK(h, concat_back(h, 8, h->dd2, h->dd3, h->de2, h->dc2, B, H / 2, W / 2));
  UCK(h, concat_back(h, 7, h->dd3, h->dbt, h->de3, h->dc3, B, H / 4, W / 4));
  // bottleneck and encoder
  UCK(h, layer_back(h, 6, h->dbt, h->dp3, nullptr, B, H / 8, W / 8, nullptr));
  k_pool_back_add<<<grid_for(pixels(B, H, W, 2) * 12), 256, 0, h->stream>>>(h->dp3, 96, B, H / 4, W / 4, h->act[5],
                                                                          h->de3);
  UCK(h, layer_back(h, 5, h->de3, h->de3a, h->act[4], B, H / 4, W / 4, nullptr));
  UCK(h, layer_back(h, 4, h->de3a, h->dp2, nullptr, B, H / 4, W / 4, nullptr));
  k_pool_back_add<<<grid_for(pixels(B, H, W, 1) * 8), 256, 0, h->stream>>>(h->dp2, 64, B, H / 2, W / 2, h->act[3],
                                                                         h->de2);
  UCK(h, layer_back(h, 3, h->de2, h->de2a, h->act[2], B, H / 2, W / 2, nullptr));
  UCK(h, layer_back(h, 2, h->de2a, h->dp1, nullptr, B, H / 2, W / 2, nullptr));
  k_pool_back_add<<<grid_for(P0 * 4), 256, 0, h->stream>>>(h->dp1, 32, B, H, W, h->act[1], h->de1);
  UCK(h, layer_back(h, 1, h->de1, h->de1a, h->act[0], B, H, W, nullptr));
  UCK(h, layer_back(h, 0, h->de1a, nullptr, nullptr, B, H, W, nullptr));
  k_reduce_few<<<FEW_SUMS, 256, 0, h->stream>>>(h->few);
  UCK(h, cudaEventRecord(h->side_done, h->side));
  UCK(h, cudaStreamWaitEvent(h->stream, h->side_done, 0));
  UCK(h, cudaGetLastError());
  if (grad_out)
    UCK(h, cudaMemcpyAsync(grad_out, h->grad, h->nparam * sizeof(float), cudaMemcpyDeviceToDevice, h->stream));
  if (loss_host) {
    UCK(h, cudaMemcpyAsync(h->sums_host, h->sums, 3 * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    UCK(h, cudaStreamSynchronize(h->stream));
    *loss_host = h->sums_host[2];
  }
  h->have_grad = true;
  return PISM_GPU_SSA_OK;
}

int pism_gpu_unet_adam(pism_gpu_unet *h, float lr, float beta1, float beta2, float eps) {
  if (!h) return PISM_GPU_SSA_EINVAL;
  if (!h->have_grad) return ufail(h, PISM_GPU_SSA_ESTATE, "adam needs a backward first");
  if (!(lr > 0.0f) || !(beta1 >= 0.0f && beta1 < 1.0f) || !(beta2 >= 0.0f && beta2 < 1.0f) || !(eps > 0.0f))
    return ufail(h, PISM_GPU_SSA_EINVAL, "adam: lr > 0, 0 <= beta < 1, eps > 0");
  UDevice dg(h->device);
  h->adam_t += 1;
  const float c1 = 1.0f - std::pow(beta1, (float)h->adam_t), c2 = 1.0f - std::pow(beta2, (float)h->adam_t);
  k_adam<<<grid_for(h->nparam), 256, 0, h->stream>>>(h->p32, h->grad, h->m, h->v, h->nparam, lr, beta1, beta2, eps, c1,
                                                      c2, h->p16);
  UCK(h, cudaGetLastError());
  return PISM_GPU_SSA_OK;
}

}  // extern "C"
