// Learned initial guess for the zeta solve: network kernels (inference and training) and the
// solver-side feature / scatter / record kernels.  Network shape and parameter layout are fixed by
// include/si3d_learn.h.
//
// Channels-last images with a one-pixel halo.  The four 32 -> 32 forward convolutions run on the
// fifth-generation tensor cores (k_conv32_tc: TMA halo loads, tcgen05.mma into TMEM, a pipeline of
// producer, MMA and epilogue warps; see there).  The data gradient for training is an implicit GEMM
// on 8 x 16 pixel tiles with mma.sync m16n8k16 (M = 16 pixels of a tile row, N = 8 channels, K = 16
// channels of one tap; 9 taps x 2 channel halves = 18 K-steps) with tap-flipped, channel-transposed
// weights.  BF16 operands, FP32 accumulation.  The 32 -> 32 weight gradients run on the tensor cores too
// (k_wgrad32: mma.sync on an exact split of the FP32 operand).  The 4 -> 32 stem, the 32 -> 1 head and
// their weight gradients are small and run on the FP32 cores, accumulating in a fixed order.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "../../include/si3d_gpu.h"
#include "../../include/si3d_learn.h"
#include "common.cuh"
#include "learn.h"

namespace si3d {
namespace learn {

namespace {

using bf16 = __nv_bfloat16;

constexpr int C = SI3D_NET_C;
constexpr int TH = 8, TW = 16, TP = TH * TW;   // pixel tile
constexpr int HT = TH + 2, WT = TW + 2;        // tile with halo
constexpr int XS = 40;                         // shared-memory pixel stride of 32-channel tiles (bf16)
constexpr int OFF_STEM_B = 9 * 4 * C;
constexpr int OFF_BLK = OFF_STEM_B + C;
constexpr int BLK_SZ = 9 * C * C + C;
constexpr int OFF_HEAD_W = OFF_BLK + SI3D_NET_BLOCKS * BLK_SZ;
constexpr int OFF_HEAD_B = OFF_HEAD_W + 9 * C;
static_assert(OFF_HEAD_B + 1 == SI3D_NET_NPARAM, "parameter layout");
constexpr int WG_BLOCKS = 296;                 // weight-gradient partial sums (2 per SM)

__device__ __forceinline__ float bfr(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// A tile of 32-channel pixels with its frame to shared memory (XS bf16 a pixel), zero outside the
// image, by asynchronous 16-byte copies: all in flight at once, without a register.  The caller waits.
template <int ROWS, int COLS, int NT>
__device__ __forceinline__ void stage_tile(bf16* sX, const bf16* __restrict__ X, int b, int i0, int j0, int H, int W) {
  for (int r = threadIdx.x; r < ROWS * COLS * 4; r += NT) {
    const int pix = r >> 2, part = r & 3;
    const int gi = i0 + pix / COLS - 1, gj = j0 + pix % COLS - 1;
    const bool in = gi >= 0 && gi < H && gj >= 0 && gj < W;
    const bf16* src = in ? X + (((size_t)b * H + gi) * W + gj) * C + part * 8 : X;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n"
                 :: "r"((uint32_t)__cvta_generic_to_shared(&sX[pix * XS + part * 8])), "l"(src), "r"(in ? 16 : 0) : "memory");
  }
}

// ------------------------------------------------------------------ weights
// Block weights to the tensor-core layout [tap][n][k] (bf16): forward n = cout, k = cin;
// data gradient n = cin, k = cout with the tap mirrored.  Stem/head weights rounded to bf16 values.
__global__ void k_prep(const float* __restrict__ prm, bf16* __restrict__ wfwd, bf16* __restrict__ wbwd,
                       float* __restrict__ stem, float* __restrict__ head) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int nb = SI3D_NET_BLOCKS * 9 * C * C;
  if (tid < nb) {
    const int blk = tid / (9 * C * C), r = tid % (9 * C * C);
    const int t = r / (C * C), n = (r / C) % C, k = r % C;
    const float* W = prm + OFF_BLK + blk * BLK_SZ;
    wfwd[tid] = __float2bfloat16_rn(W[(t * C + k) * C + n]);          // W[t][cin=k][cout=n]
    wbwd[tid] = __float2bfloat16_rn(W[((8 - t) * C + n) * C + k]);    // W[8-t][cin=n][cout=k]
  }
  if (tid < 9 * 4 * C) stem[tid] = bfr(prm[tid]);
  if (tid < C) stem[9 * 4 * C + tid] = prm[OFF_STEM_B + tid];
  if (tid < 9 * C) head[tid] = bfr(prm[OFF_HEAD_W + tid]);
  if (tid == 0) head[9 * C] = prm[OFF_HEAD_B];
}

// ------------------------------------------------------------------ stem: 4 -> 32, FP32 cores
// A block takes 8 rows x 32 pixels, a warp a row, a lane an output channel with its 36 weights in
// registers.  The warp walks the row with the 3 x 3 window of the input (four channels each, the same for
// all lanes) in registers, so a pixel costs three 16-byte broadcasts for 36 FMA, and a pixel's 32
// channels are stored side by side.  Per output channel the products are accumulated in the order tap,
// input channel, with the inputs rounded to BF16 first.  Weights from shared memory, a thread all channels
// of two pixels: 80 us at 1002 x 502 pixels; this: 42 (of which 24 are instruction issue; two pixels'
// chains interleaved 52, three blocks an SM 43, persistent blocks with the next tile fetched ahead 45).
constexpr int ST_W = 2 * TW;                   // pixels per row of a stem tile
constexpr int ST_WT = ST_W + 2;                // with halo
__global__ void __launch_bounds__(32 * TH) k_stem(const float* __restrict__ feat, const float* __restrict__ w, int H, int W,
                                                  bf16* __restrict__ X, float* __restrict__ Y) {
  __shared__ __align__(16) float sF[HT * ST_WT * 4];
  const int b = blockIdx.z, i0 = blockIdx.y * TH, j0 = blockIdx.x * ST_W;
  const int co = threadIdx.x & 31, ti = threadIdx.x >> 5;
  float wr[36];
#pragma unroll
  for (int t = 0; t < 36; ++t) wr[t] = w[t * C + co];
  const float bias = w[36 * C + co];
  for (int r = threadIdx.x; r < HT * ST_WT; r += 32 * TH) {
    const int gi = i0 + r / ST_WT - 1, gj = j0 + r % ST_WT - 1;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (gi >= 0 && gi < H && gj >= 0 && gj < W) v = *reinterpret_cast<const float4*>(feat + (((size_t)b * H + gi) * W + gj) * 4);
    *reinterpret_cast<float4*>(&sF[r * 4]) = make_float4(bfr(v.x), bfr(v.y), bfr(v.z), bfr(v.w));
  }
  __syncthreads();
  const int gi = i0 + ti;
  if (gi >= H) return;
  const size_t p0 = ((size_t)b * H + gi) * W + j0;
  const int n = min(ST_W, W - j0);
  float4 x[3][3];   // rows, columns of the window
  auto column = [&](int c, int tj) {
#pragma unroll
    for (int i = 0; i < 3; ++i) x[i][c] = *reinterpret_cast<const float4*>(&sF[((ti + i) * ST_WT + tj) * 4]);
  };
  column(0, 0);
  column(1, 1);
#pragma unroll 4
  for (int tj = 0; tj < n; ++tj) {
    column(2, tj + 2);
    float acc = 0.f;
#pragma unroll
    for (int t = 0; t < 9; ++t) {
      const float4 v = x[t / 3][t % 3];
      acc = __fmaf_rn(v.x, wr[4 * t], acc);
      acc = __fmaf_rn(v.y, wr[4 * t + 1], acc);
      acc = __fmaf_rn(v.z, wr[4 * t + 2], acc);
      acc = __fmaf_rn(v.w, wr[4 * t + 3], acc);
    }
    const float y = acc + bias;
    const size_t o = (p0 + tj) * C + co;
    if (Y) Y[o] = y;
    X[o] = __float2bfloat16_rn(fmaxf(y, 0.f));
#pragma unroll
    for (int i = 0; i < 3; ++i) { x[i][0] = x[i][1]; x[i][1] = x[i][2]; }
  }
}

// ------------------------------------------------------------------ 32 -> 32 conv on the tensor cores
__device__ __forceinline__ void mma_bf16(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Behind a layer's G (the gradient of its input x_k): DY = G * (y_k > 0), the gradient at the ReLU of
// the layer below, in FP32 for the weight gradient and (unless it is the stem's) in BF16 for the
// tensor-core data gradient.  Written by the kernel that makes G, which spares a pass over G a layer
// (32 x 64 x 64 pixels: five passes of 19.5 us against 7 us more in the data gradient).
__device__ __forceinline__ float relu_grad(float g, float y) { return y > 0.f ? g : 0.f; }

// Data gradient of a 32 -> 32 layer: G[p][n] += sum_{tap, k} in[p + off(tap)][k] * Wk[tap][n][k], in place
// (a thread reads and writes the same elements), and for the layer below DY and (not for the stem) DYb
// from its y.  Persistent blocks: the weights go to shared memory once per block, which then loops over
// 8 x 16 pixel tiles (tile = blockIdx.x, blockIdx.x + gridDim.x, ...).  Tiles by asynchronous copies and a
// row's G and Y loaded together: 32.6 -> 26.4 us at 32 x 64 x 64 pixels (84 MB: 13 us at memory's rate).
__global__ void __launch_bounds__(128) k_conv32_bwd(const bf16* __restrict__ Xin, const bf16* __restrict__ Wk, int B,
                                                    int H, int W, float* __restrict__ G, const float* __restrict__ Y,
                                                    float* __restrict__ DY, bf16* __restrict__ DYb) {
  __shared__ __align__(16) bf16 sX[HT * WT * XS];
  __shared__ __align__(16) bf16 sW[9 * C * XS];
  for (int r = threadIdx.x; r < 9 * C * 4; r += 128) {
    const int row = r >> 2, part = r & 3;
    *reinterpret_cast<uint4*>(&sW[row * XS + part * 8]) = *reinterpret_cast<const uint4*>(&Wk[row * C + part * 8]);
  }
  const int ntj = (W + TW - 1) / TW, nti = (H + TH - 1) / TH, ntiles = B * nti * ntj;
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int b = tile / (nti * ntj), rem = tile - b * (nti * ntj);
    const int i0 = (rem / ntj) * TH, j0 = (rem % ntj) * TW;
    __syncthreads();   // the previous tile's readers of sX are done
    stage_tile<HT, WT, 128>(sX, Xin, b, i0, j0, H, W);
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    float acc[2][4][4];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[r][nt][e] = 0.f;
#pragma unroll 1
    for (int t = 0; t < 9; ++t) {
      const int di = t / 3 - 1, dj = t % 3 - 1;
#pragma unroll
      for (int cb = 0; cb < 2; ++cb) {
        uint32_t bq[4][2];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          const bf16* wp = &sW[(t * C + nt * 8 + g) * XS + cb * 16 + q * 2];
          bq[nt][0] = *reinterpret_cast<const uint32_t*>(wp);
          bq[nt][1] = *reinterpret_cast<const uint32_t*>(wp + 8);
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int ty = warp * 2 + r;
          const bf16* xp = &sX[((ty + 1 + di) * WT + (g + 1 + dj)) * XS + cb * 16 + q * 2];
          const uint32_t a0 = *reinterpret_cast<const uint32_t*>(xp);
          const uint32_t a1 = *reinterpret_cast<const uint32_t*>(xp + 8 * XS);
          const uint32_t a2 = *reinterpret_cast<const uint32_t*>(xp + 8);
          const uint32_t a3 = *reinterpret_cast<const uint32_t*>(xp + 8 * XS + 8);
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) mma_bf16(acc[r][nt], a0, a1, a2, a3, bq[nt][0], bq[nt][1]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int gi = i0 + warp * 2 + r;
      if (gi >= H) continue;
      const size_t o0 = (((size_t)b * H + gi) * W + j0) * C + 2 * q;
      float2 gin[2][4], y[2][4];   // the row's values, all loads in flight at once
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int tj = g + 8 * half;
        if (j0 + tj < W) {
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) {
            gin[half][nt] = *reinterpret_cast<const float2*>(G + o0 + tj * C + nt * 8);
            y[half][nt] = *reinterpret_cast<const float2*>(Y + o0 + tj * C + nt * 8);
          }
        }
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int tj = g + 8 * half;
        if (j0 + tj >= W) continue;
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          const size_t o = o0 + tj * C + nt * 8;
          const float2 go = make_float2(gin[half][nt].x + acc[r][nt][2 * half], gin[half][nt].y + acc[r][nt][2 * half + 1]);
          const float2 d = make_float2(relu_grad(go.x, y[half][nt].x), relu_grad(go.y, y[half][nt].y));
          *reinterpret_cast<float2*>(DY + o) = d;
          if (DYb) {
            *reinterpret_cast<float2*>(G + o) = go;
            *reinterpret_cast<__nv_bfloat162*>(DYb + o) = __floats2bfloat162_rn(d.x, d.y);
          }
        }
      }
    }
  }
}

// ------------------------------------------------------------------ 32 -> 32 conv, tcgen05 (forward)
// The convolution on the fifth-generation tensor cores, as a pipeline in one persistent block per
// SM that walks tiles of TC_R output rows x 128 pixels (tile blockIdx.x, + gridDim.x, ...):
//   warp 0 (one lane)   loads each tile's halo (TC_R + 2 rows x 130 pixels x 32 bf16 channels) with
//                       four TMA copies, one per 8-channel chunk, into a ring of TC_NS stages,
//                       zero-filled outside the image;
//   warp 1 (one lane)   issues per output row 9 taps x 2 K-halves = 18 tcgen05.mma (M = 128
//                       pixels, N = 32, K = 16, BF16 in, FP32 accumulate) into that row's 32 columns
//                       of one of two TMEM accumulators, then commits to the accumulator's "full"
//                       barrier and to the stage's "empty" barrier;
//   warps 2-17          read the accumulator (each warp its 32 TMEM lanes, i.e. pixels, of its row), add bias,
//                       ReLU and the residual (from the same stage), store, and release the
//                       accumulator and the stage.
// So tile i + 1 loads and tile i multiplies while tile i - 1 is written.  Four warps a row of the tile
// write it: four warps in all could not hide the latency of their own chain (TMEM, shared memory, global
// memory), and leaving out the loads, the multiplications or the stores changed the time by less than
// a tenth.  A call at 1002 x 502 pixels 70 -> 38 us, at 32 x 64 x 64 with Y 29 -> 21 us (ncu).  The stage holds
// [chunk][row][pixel][8 channels]: the A operand of tap (di, dj) for output row r is a K-major
// no-swizzle matrix starting at row r + 1 + di, pixel 1 + dj (core matrices of 8 pixels x 16 bytes,
// 128 bytes between pixel groups, one chunk between K halves) - no im2col.  Weights sit as
// sB[tap][chunk][cout][8 cin].  Every mbarrier wait is bounded; a role whose wait gives up raises a
// flag the others see, and the epilogue then writes NaN into the tiles it has not written, which
// the solve rejects.
constexpr int TC_R = 4;                        // output rows per tile
constexpr int TC_W = 128;                      // pixels per row (the MMA's M)
constexpr int TC_WT = TC_W + 2;                // with halo
constexpr int TC_CHUNK_TX = (TC_R + 2) * TC_WT * 16;   // bytes one chunk's TMA copy writes (12,480)
constexpr int TC_CHUNK = (TC_CHUNK_TX + 127) / 128 * 128;   // chunk stride, 128-byte aligned (12,544)
constexpr int TC_ROWB = TC_WT * 16;            // bytes of one halo row of a chunk
constexpr int TC_STAGE = 4 * TC_CHUNK;         // one halo tile
constexpr int TC_NS = 3;                       // halo tiles in flight
constexpr int TC_BBYTES = 9 * 4 * C * 16;      // 18,432
constexpr int TC_OSTRIDE = 80;                 // bytes per pixel of an epilogue warp's staging rows (64 + 16)
constexpr int TC_EW = 4 * TC_R;                // epilogue warps: four a row
constexpr int TC_OBYTES = TC_EW * 32 * TC_OSTRIDE;   // 32 pixels each
constexpr int TC_SMEM = TC_NS * TC_STAGE + TC_BBYTES + TC_OBYTES + 1024;   // + alignment of the dynamic base
constexpr int TC_ACC = TC_R * C;               // TMEM columns of one accumulator (128)
constexpr int TC_COLS = 2 * TC_ACC;            // two accumulators
constexpr int TC_THREADS = 64 + 32 * TC_EW;
constexpr long long TC_WAIT_LIMIT = 1LL << 24; // mbarrier polls before giving up
static_assert(TC_COLS == 256, "TMEM allocation");
static_assert(TC_STAGE % 1024 == 0 || TC_CHUNK % 128 == 0, "TMA destinations 128-byte aligned");

// Instruction descriptor of kind::f16: D FP32, A and B BF16, both K-major, N = 32, M = 128.
constexpr uint32_t TC_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(C >> 3) << 17) | ((uint32_t)(TC_W >> 4) << 24);

// Shared-memory matrix descriptor, no swizzle: start address, the byte offsets between core
// matrices along K (leading) and along M/N (stride), descriptor version 1.
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Bounded wait for the completion of phase `parity` of an mbarrier; gives up (raising *fail) after
// TC_WAIT_LIMIT polls, or at once when another role has raised *fail.
__device__ __forceinline__ bool tc_wait(uint32_t mbar, uint32_t parity, volatile int* fail, bool heed = true) {
  for (long long it = 0; it < TC_WAIT_LIMIT; ++it) {
    uint32_t ok;
    asm volatile("{\n.reg .pred q;\nmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\nselp.u32 %0, 1, 0, q;\n}\n"
                 : "=r"(ok) : "r"(mbar), "r"(parity) : "memory");
    if (ok) return true;
    if (heed && (it & 63) == 0 && *fail) return false;
  }
  *fail = 1;
  return false;
}

__device__ __forceinline__ void tc_arrive(uint32_t mbar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" :: "r"(mbar) : "memory");
}

__global__ void __launch_bounds__(TC_THREADS, 1) k_conv32_tc(const __grid_constant__ CUtensorMap xmap,
                                                             const bf16* __restrict__ Wk,
                                                             const float* __restrict__ bias, int B, int H, int W,
                                                             bf16* __restrict__ Xout, float* __restrict__ Y) {
  extern __shared__ unsigned char smem_raw[];
  __shared__ uint32_t s_tmem;
  __shared__ __align__(8) unsigned long long s_bar[2 * TC_NS + 4];   // full[NS], empty[NS], tfull[2], tempty[2]
  __shared__ __align__(16) float s_bias[C];
  __shared__ volatile int s_fail;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rawBase = (uint32_t)__cvta_generic_to_shared(smem_raw);
  const uint32_t aBase = (rawBase + 1023u) & ~1023u;              // TC_NS stages of TC_STAGE bytes
  const uint32_t bBase = aBase + TC_NS * TC_STAGE;
  unsigned char* const sA = smem_raw + (aBase - rawBase);
  unsigned char* const sB = smem_raw + (bBase - rawBase);
  const uint32_t bar0 = (uint32_t)__cvta_generic_to_shared(&s_bar[0]);
  auto full = [&](int st) { return bar0 + 8u * (uint32_t)st; };
  auto empty = [&](int st) { return bar0 + 8u * (uint32_t)(TC_NS + st); };
  auto tfull = [&](int a) { return bar0 + 8u * (uint32_t)(2 * TC_NS + a); };
  auto tempty = [&](int a) { return bar0 + 8u * (uint32_t)(2 * TC_NS + 2 + a); };
  // weights -> sB[tap][chunk][cout][8], bias; barriers; TMEM (warp 1)
  for (int r = tid; r < 9 * C * 4; r += TC_THREADS) {
    const int t = r / (C * 4), n = (r / 4) % C, kc = r % 4;
    *reinterpret_cast<uint4*>(sB + (((t * 4 + kc) * C + n) * 16)) =
        *reinterpret_cast<const uint4*>(&Wk[(t * C + n) * C + kc * 8]);
  }
  for (int r = tid; r < C; r += TC_THREADS) s_bias[r] = bias[r];
  if (tid == 0) {
    s_fail = 0;
    for (int st = 0; st < TC_NS; ++st) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" :: "r"(full(st)) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n"
                   :: "r"(empty(st)), "r"(1 + TC_EW) : "memory");   // commit + the epilogue's warps
    }
    for (int a = 0; a < 2; ++a) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" :: "r"(tfull(a)) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" :: "r"(tempty(a)), "r"(TC_EW) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("prefetch.tensormap [%0];\n" :: "l"(reinterpret_cast<uint64_t>(&xmap)) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                 :: "r"((uint32_t)__cvta_generic_to_shared(&s_tmem)), "r"((uint32_t)TC_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  // the weights (generic-proxy writes) become visible to the tensor core's reads
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = s_tmem;
  const int ntj = (W + TC_W - 1) / TC_W, nti = (H + TC_R - 1) / TC_R, ntiles = B * nti * ntj;
  auto tile_origin = [&](int t, int& b, int& i0, int& j0) {
    b = t / (nti * ntj);
    const int rem = t - b * (nti * ntj);
    i0 = (rem / ntj) * TC_R;
    j0 = (rem % ntj) * TC_W;
  };
  if (warp == 0) {
    // ---------------------------------------------------------------- producer
    if (lane == 0) {
      int issued = 0;
      for (int i = 0, t = blockIdx.x; t < ntiles; ++i, t += gridDim.x) {
        const int st = i % TC_NS;
        if (i >= TC_NS && !tc_wait(empty(st), (uint32_t)((i / TC_NS - 1) & 1), &s_fail)) break;
        issued = i + 1;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n"
                     :: "r"(full(st)), "r"((uint32_t)(4 * TC_CHUNK_TX)) : "memory");
        int b, i0, j0;
        tile_origin(t, b, i0, j0);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint32_t dst = aBase + (uint32_t)(st * TC_STAGE + c * TC_CHUNK);
          asm volatile(
              "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n"
              :: "r"(dst), "l"(reinterpret_cast<uint64_t>(&xmap)), "r"(c * 8), "r"(j0 - 1), "r"(i0 - 1), "r"(b),
                 "r"(full(st)) : "memory");
        }
      }
      // after a failure, the copies still in flight land before the block leaves
      if (s_fail)
        for (int i = (issued > TC_NS ? issued - TC_NS : 0); i < issued; ++i)
          tc_wait(full(i % TC_NS), (uint32_t)((i / TC_NS) & 1), &s_fail, false);
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issue
    if (lane == 0) {
      int issued = 0;
      for (int i = 0, t = blockIdx.x; t < ntiles; ++i, t += gridDim.x) {
        const int st = i % TC_NS, a = i & 1;
        if (!tc_wait(full(st), (uint32_t)((i / TC_NS) & 1), &s_fail)) break;
        if (i >= 2 && !tc_wait(tempty(a), (uint32_t)((i / 2 - 1) & 1), &s_fail)) break;
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        // descriptors of the stage's first A matrix and of the first B matrix; the other 71 differ only
        // in their start address (the low 14 bits, address / 16), by compile-time offsets, so the
        // fully unrolled issue is an add and an MMA each
        const uint64_t ad0 = tc_desc(aBase + (uint32_t)(st * TC_STAGE), TC_CHUNK, 128);
        const uint64_t bd0 = tc_desc(bBase, C * 16, 128);
        const uint32_t d0 = tmem + (uint32_t)(a * TC_ACC);
#pragma unroll
        for (int r = 0; r < TC_R; ++r) {
#pragma unroll
          for (int tap = 0; tap < 9; ++tap) {
            const int di = tap / 3 - 1, dj = tap % 3 - 1;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const uint64_t ad = ad0 + (uint64_t)((2 * h * TC_CHUNK + (r + 1 + di) * TC_ROWB + (1 + dj) * 16) >> 4);
              const uint64_t bd = bd0 + (uint64_t)((((tap * 4 + 2 * h) * C) * 16) >> 4);
              const uint32_t acc = (tap > 0 || h > 0) ? 1u : 0u;   // the row's first product starts it
              asm volatile(
                  "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                  "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                  :: "r"(d0 + (uint32_t)(r * C)), "l"(ad), "l"(bd), "r"(TC_IDESC), "r"(acc) : "memory");
            }
          }
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
                     :: "r"(tfull(a)) : "memory");
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
                     :: "r"(empty(st)) : "memory");
        ++issued;
      }
      // the last multiplications have finished before the accumulators are freed
      if (issued > 0) tc_wait(tfull((issued - 1) & 1), (uint32_t)(((issued - 1) / 2) & 1), &s_fail);
    }
  } else {
    // ---------------------------------------------------------------- epilogue (warps 2-17)
    const int q = warp & 3, r = (warp - 2) >> 2;   // TMEM lanes 32 q .. 32 q + 31 = pixels of this warp; its row
    const int px = q * 32 + lane;
    // staging rows of this warp's output: the stores to global memory go out as contiguous runs
    unsigned char* const sO = sB + TC_BBYTES + (warp - 2) * 32 * TC_OSTRIDE;
    bool ok = true;
    for (int i = 0, t = blockIdx.x; t < ntiles; ++i, t += gridDim.x) {
      const int st = i % TC_NS, a = i & 1;
      int b, i0, j0;
      tile_origin(t, b, i0, j0);
      // one lane of the warp waits (the others would only compete with the tensor core for shared
      // memory) for the accumulator and for the stage's halo tile, which is read below for the
      // residual (its barrier is complete already: the stage cannot be refilled before this warp
      // releases it); __syncwarp orders the other lanes' reads after the wait
      if (lane == 0 && ok) {
        ok = tc_wait(tfull(a), (uint32_t)((i / 2) & 1), &s_fail);
        if (ok) ok = tc_wait(full(st), (uint32_t)((i / TC_NS) & 1), &s_fail);
      }
      ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;   // the TMEM reads below are warp-collective
      __syncwarp();
      if (ok) asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      const int gi = i0 + r;
      const bool row = gi < H;   // warp-uniform: otherwise the whole row is outside the image
      uint32_t v[C];
      if (ok) {
        const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(a * TC_ACC + r * C);
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
            "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
              "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
              "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
              "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
            : "r"(taddr) : "memory");
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
      } else {
#pragma unroll
        for (int k = 0; k < C; ++k) v[k] = 0u;
      }
      // the stage's values of this pixel; the accumulator and (after these) the stage are given back below
      const unsigned char* xc = sA + st * TC_STAGE + (r + 1) * TC_ROWB + (px + 1) * 16;
      const size_t p0 = ((size_t)b * H + gi) * W + (j0 + q * 32);
      if (row) {
        float y[C];
#pragma unroll
        for (int c4 = 0; c4 < C / 4; ++c4) {
          const float4 bi = *reinterpret_cast<const float4*>(&s_bias[4 * c4]);
          y[4 * c4] = __uint_as_float(v[4 * c4]) + bi.x;
          y[4 * c4 + 1] = __uint_as_float(v[4 * c4 + 1]) + bi.y;
          y[4 * c4 + 2] = __uint_as_float(v[4 * c4 + 2]) + bi.z;
          y[4 * c4 + 3] = __uint_as_float(v[4 * c4 + 3]) + bi.w;
        }
        if (!ok) {
#pragma unroll
          for (int k = 0; k < C; ++k) y[k] = __int_as_float(0x7fc00000);
        }
        // Through the staging rows a warp writes 16 bytes a lane: run k, lane l: pixel 8 k + l / 4 and the
        // l % 4-th 16 bytes of the 64 that were staged for it (X: its 32 channels, Y: half of them)
        auto flush = [&](unsigned char* out, int stride) {
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int pl = k * 8 + (lane >> 2), cc = lane & 3;
            if (j0 + q * 32 + pl < W)
              *reinterpret_cast<uint4*>(out + (p0 + pl) * (size_t)stride + cc * 16) =
                  *reinterpret_cast<const uint4*>(sO + pl * TC_OSTRIDE + cc * 16);
          }
          __syncwarp();
        };
        if (Y) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
              *reinterpret_cast<float4*>(sO + lane * TC_OSTRIDE + k * 16) =
                  make_float4(y[h * 16 + 4 * k], y[h * 16 + 4 * k + 1], y[h * 16 + 4 * k + 2], y[h * 16 + 4 * k + 3]);
            flush(reinterpret_cast<unsigned char*>(Y) + h * 64, C * (int)sizeof(float));
          }
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint4 xin = ok ? *reinterpret_cast<const uint4*>(xc + c * TC_CHUNK) : make_uint4(0u, 0u, 0u, 0u);
          const __nv_bfloat162* x2 = reinterpret_cast<const __nv_bfloat162*>(&xin);
          uint4 o;
          uint32_t* o32 = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int co = c * 8 + 2 * e;
            const float2 xf = __bfloat1622float2(x2[e]);
            const __nv_bfloat162 ob = __floats2bfloat162_rn(xf.x + fmaxf(y[co], 0.f), xf.y + fmaxf(y[co + 1], 0.f));
            o32[e] = ok ? *reinterpret_cast<const uint32_t*>(&ob) : 0x7fc07fc0u;   // (ReLU makes 0 of a NaN)
          }
          *reinterpret_cast<uint4*>(sO + lane * TC_OSTRIDE + c * 16) = o;
        }
        flush(reinterpret_cast<unsigned char*>(Xout), C * (int)sizeof(bf16));
      }
      // this warp is done with the accumulator and the stage
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncwarp();
      if (ok && lane == 0) {
        tc_arrive(tempty(a));
        tc_arrive(empty(st));
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" :: "r"(tmem), "r"((uint32_t)TC_COLS)
                 : "memory");
  }
}

// ------------------------------------------------------------------ head: 32 -> 1, FP32 cores
// A thread computes four pixels of a column (tile: 8 rows x 32 pixels): a value of X read from shared
// memory and widened serves three rows of taps, a weight four pixels.  The products of an output are
// accumulated in the order tap column, eight channels, tap row.  A pixel a thread 31 us at 1002 x 502
// pixels; this with plain loads for the tile 29, with asynchronous copies 22.
constexpr int HD_R = 4;                        // pixels of a thread
constexpr int HD_T = TH / HD_R * ST_W;         // threads
__global__ void __launch_bounds__(HD_T) k_head(const bf16* __restrict__ X, const float* __restrict__ w, int H, int W,
                                               float* __restrict__ out) {
  __shared__ __align__(16) bf16 sX[HT * ST_WT * XS];
  __shared__ __align__(16) float sW[9 * C + 1];
  const int b = blockIdx.z, i0 = blockIdx.y * TH, j0 = blockIdx.x * ST_W;
  for (int r = threadIdx.x; r < 9 * C + 1; r += HD_T) sW[r] = w[r];
  stage_tile<HT, ST_WT, HD_T>(sX, X, b, i0, j0, H, W);
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  __syncthreads();
  const int t0 = threadIdx.x / ST_W * HD_R, tj = threadIdx.x % ST_W, gj = j0 + tj;
  if (gj >= W) return;
  float acc[HD_R];
#pragma unroll
  for (int i = 0; i < HD_R; ++i) acc[i] = 0.f;
  for (int dj = 0; dj < 3; ++dj) {
#pragma unroll
    for (int q = 0; q < C / 8; ++q) {
      float wv[3][8];
#pragma unroll
      for (int di = 0; di < 3; ++di) {
        const float4* w4 = reinterpret_cast<const float4*>(&sW[(di * 3 + dj) * C + 8 * q]);
        const float4 a = w4[0], c = w4[1];
        wv[di][0] = a.x; wv[di][1] = a.y; wv[di][2] = a.z; wv[di][3] = a.w;
        wv[di][4] = c.x; wv[di][5] = c.y; wv[di][6] = c.z; wv[di][7] = c.w;
      }
#pragma unroll
      for (int i = 0; i < HD_R + 2; ++i) {   // halo rows: row i is tap row di of pixel i - di
        const uint4 xv = *reinterpret_cast<const uint4*>(&sX[((t0 + i) * ST_WT + tj + dj) * XS + 8 * q]);
        const __nv_bfloat162* x2 = reinterpret_cast<const __nv_bfloat162*>(&xv);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 f = __bfloat1622float2(x2[e]);
#pragma unroll
          for (int di = 0; di < 3; ++di)
            if (i - di >= 0 && i - di < HD_R) {
              acc[i - di] = __fmaf_rn(f.x, wv[di][2 * e], acc[i - di]);
              acc[i - di] = __fmaf_rn(f.y, wv[di][2 * e + 1], acc[i - di]);
            }
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < HD_R; ++i)
    if (i0 + t0 + i < H) out[((size_t)b * H + i0 + t0 + i) * W + gj] = acc[i] + sW[9 * C];
}

// ------------------------------------------------------------------ backward pieces
// G4[p][ci] = sum_tap gout[p - off(tap)] * wh[tap][ci], and DY, DYb from it.  A thread has four channels
// of a pixel, so that a warp writes whole lines (29 -> 15 us at 32 x 64 x 64, the ReLU's pass included).
__global__ void __launch_bounds__(TP) k_head_bwd(const float* __restrict__ gout, const float* __restrict__ w, int H,
                                                 int W, const float* __restrict__ Y, float* __restrict__ G,
                                                 float* __restrict__ DY, bf16* __restrict__ DYb) {
  __shared__ float sG[HT * WT];
  const int b = blockIdx.z, i0 = blockIdx.y * TH, j0 = blockIdx.x * TW;
  const int c4 = (threadIdx.x % (C / 4)) * 4;
  float wr[9][4];
#pragma unroll
  for (int t = 0; t < 9; ++t)
#pragma unroll
    for (int e = 0; e < 4; ++e) wr[t][e] = w[t * C + c4 + e];
  for (int r = threadIdx.x; r < HT * WT; r += TP) {
    const int gi = i0 + r / WT - 1, gj = j0 + r % WT - 1;
    sG[r] = (gi >= 0 && gi < H && gj >= 0 && gj < W) ? gout[((size_t)b * H + gi) * W + gj] : 0.f;
  }
  __syncthreads();
#pragma unroll 4
  for (int pix = threadIdx.x / (C / 4); pix < TP; pix += TP / (C / 4)) {
    const int ti = pix / TW, tj = pix % TW, gi = i0 + ti, gj = j0 + tj;
    if (gi >= H || gj >= W) continue;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int t = 0; t < 9; ++t) {
      const int tm = 8 - t;   // gout at p + off(8 - t) = p - off(t)
      const float g = sG[(ti + tm / 3) * WT + tj + tm % 3];
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[e] = acc[e] + g * wr[t][e];
    }
    const size_t o = (((size_t)b * H + gi) * W + gj) * C + c4;
    const float4 y = *reinterpret_cast<const float4*>(Y + o);
    const float4 d = make_float4(relu_grad(acc[0], y.x), relu_grad(acc[1], y.y), relu_grad(acc[2], y.z), relu_grad(acc[3], y.w));
    *reinterpret_cast<float4*>(G + o) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    *reinterpret_cast<float4*>(DY + o) = d;
    *reinterpret_cast<__nv_bfloat162*>(DYb + o) = __floats2bfloat162_rn(d.x, d.y);
    *reinterpret_cast<__nv_bfloat162*>(DYb + o + 2) = __floats2bfloat162_rn(d.z, d.w);
  }
}

// Weight gradient partials: part[blk][(tap * CIN + ci) * COUT + co] = sum over the block's tiles of
// X[p + off(tap)][ci] * DY[p][co], and part[blk][9 * CIN * COUT + co] = sum DY[p][co].
constexpr int GH = 4, GP = GH * TW;        // tiles: 4 x 16 pixels
constexpr int GHP = (GH + 2) * WT;         // with frame

// 32 -> 32.  X is BF16 and DY FP32.  DY is cut into three BF16 terms of eight bits each, whose sum is DY
// exactly, so the tensor cores form the same products as FP32 multiply-adds, X * DY, and sum them in
// FP32.  A warp has one tap: M = 32 ci, N = 32 co, K = 16 pixels of a row, A and B by transposed
// ldmatrix from pixel-major tiles (80 bytes a pixel: no bank conflicts).  The next tile's X (cp.async)
// and DY (registers) are under way behind the multiplications.  The tensor core cuts where an FP32 add
// rounds, so its sums are kept short: 16 pixels of a row, three products, then an FP32 add to the
// thread's sums.  Error against 64 bits (relative, L2 over the gradient; six cases of 128 to 131,072
// pixels): 0.7e-7 to 1.7e-7, of FP32 multiply-adds 1.1e-7 to 3.9e-7; with one chain a tile or a block it
// would be up to 3 times that of FP32.  32 x 64 x 64 pixels, per call: FP32 cores, one load a multiply-add
// 200 us; FP32 cores, 9 x 4 sums a thread 66 (9 x 8: 67, packed pairs: 65; bound by the FP32 pipes); this: 32.
// Two kinds of values need more, and a block that meets one walks its tiles a second time in the WIDE form
// (looking out for them takes 1.7 us a call, the WIDE form at once would take 7.5 us):
//   a DY below kTiny, whose lower terms would fall below BF16's range: in the WIDE form a term is held 2^7
//   times as large as its part of DY, once for the second and twice for the third, and the sums are scaled
//   back between the terms.  2^7 and no more, so that no term is larger than the one before;
//   an infinite X, which gives NaN against a lower term that is zero where DY is not: in the WIDE form the
//   lower terms meet X without its infinities.  (The lower terms of an infinite DY are zero.)
constexpr int GT = 9 * 32;                 // threads: a warp a tap
__device__ __forceinline__ void ldsm4t(uint32_t* r, const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ uint32_t top_halves(float a, float b) {   // two FP32 cut to BF16, a in the low half
  return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}
__device__ __forceinline__ float cut(float a) { return __uint_as_float(__float_as_uint(a) & 0xffff0000u); }
__device__ __forceinline__ float rest(float a) { return isinf(a) ? 0.f : a - cut(a); }   // exact
constexpr uint32_t kTiny = (127u - 100u) << 23;   // 2^-100: its third term's last bit is 2^-123, a normal number
__device__ __forceinline__ uint32_t magnitude(float a) { return (__float_as_uint(a) << 1) - 1u; }   // zero: the largest

__global__ void __launch_bounds__(GT, 2) k_wgrad32(const bf16* __restrict__ X, const float* __restrict__ DY, int B, int H,
                                                   int W, float* __restrict__ part) {
  __shared__ __align__(16) bf16 sX[2][GHP * XS];
  __shared__ __align__(16) bf16 sD[3][GP * XS];
  constexpr int ND = (GP * C / 4 + GT - 1) / GT;   // float4 of DY a thread stages
  const int ln = threadIdx.x & 31, tap = threadIdx.x >> 5;
  const int nj = (W + TW - 1) / TW, ni = (H + GH - 1) / GH, ntiles = B * ni * nj;
  const int c4 = threadIdx.x % (C / 4) * 4;        // the channels it stages (GT is a multiple of 8)
  float acc[2][4][4];                              // [ci / 16][co / 8][fragment]
  float4 sum, rd[ND];
  auto fetch = [&](int tile, int buf) {
    const int b = tile / (ni * nj), rem = tile - b * (ni * nj), i0 = rem / nj * GH, j0 = rem % nj * TW;
    stage_tile<GH + 2, WT, GT>(sX[buf], X, b, i0, j0, H, W);
#pragma unroll
    for (int k = 0; k < ND; ++k) {
      const int pix = (threadIdx.x + k * GT) / (C / 4), gi = i0 + pix / TW, gj = j0 + pix % TW;
      rd[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (pix < GP && gi < H && gj < W)
        rd[k] = *reinterpret_cast<const float4*>(DY + (((size_t)b * H + gi) * W + gj) * C + c4);
    }
  };
  auto walk = [&](auto form) -> bool {   // whether it met a value that needs the WIDE form
    constexpr bool WIDE = decltype(form)::value;
    uint32_t least = 0xffffffffu;
    int buf = 0;
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int n = 0; n < 4; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[m][n][e] = 0.f;
    sum = make_float4(0.f, 0.f, 0.f, 0.f);
    if ((int)blockIdx.x < ntiles) fetch(blockIdx.x, 0);
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, buf ^= 1) {
      __syncthreads();   // the previous tile's readers are done
#pragma unroll
      for (int k = 0; k < ND; ++k) {
        const int pix = (threadIdx.x + k * GT) / (C / 4);
        float4 d = rd[k];
        sum.x = sum.x + d.x; sum.y = sum.y + d.y; sum.z = sum.z + d.z; sum.w = sum.w + d.w;
        if (!WIDE) least = min(min(least, min(magnitude(d.x), magnitude(d.y))), min(magnitude(d.z), magnitude(d.w)));
        if (pix < GP) {
#pragma unroll
          for (int s = 0; s < 3; ++s) {
            *reinterpret_cast<uint2*>(&sD[s][pix * XS + c4]) = make_uint2(top_halves(d.x, d.y), top_halves(d.z, d.w));
            const float up = WIDE ? 128.f : 1.f;
            d = make_float4(up * rest(d.x), up * rest(d.y), up * rest(d.z), up * rest(d.w));
          }
        }
      }
      asm volatile("cp.async.wait_all;\n" ::: "memory");
      __syncthreads();
      if (tile + (int)gridDim.x < ntiles) fetch(tile + gridDim.x, buf ^ 1);
      const bf16* xa = &sX[buf][((tap / 3) * WT + tap % 3 + (ln & 7) + (ln >> 4) * 8) * XS + ((ln >> 3) & 1) * 8];
      const int ob = ((ln & 7) + ((ln >> 3) & 1) * 8) * XS + (ln >> 4) * 8;
#pragma unroll
      for (int ti = 0; ti < GH; ++ti) {
        uint32_t a[2][4];
        ldsm4t(a[0], xa + ti * WT * XS);
        ldsm4t(a[1], xa + ti * WT * XS + 16);
        auto lower = [&](uint32_t x) {   // X for the lower terms
          return WIDE ? x & ~__vcmpeq2(x & 0x7fff7fffu, 0x7f807f80u) : x;
        };
#pragma unroll
        for (int n2 = 0; n2 < 2; ++n2) {
          float r[2][2][4];   // the sums over this row's 16 pixels
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int e = 0; e < 4; ++e) r[m][0][e] = r[m][1][e] = 0.f;
#pragma unroll
          for (int s = 2; s >= 0; --s) {   // the small terms first
            uint32_t bq[4];
            ldsm4t(bq, &sD[s][ti * TW * XS + ob + n2 * 16]);
#pragma unroll
            for (int m = 0; m < 2; ++m) {
              uint32_t x[4];
#pragma unroll
              for (int e = 0; e < 4; ++e) x[e] = s > 0 ? lower(a[m][e]) : a[m][e];
              mma_bf16(r[m][0], x[0], x[1], x[2], x[3], bq[0], bq[1]);
              mma_bf16(r[m][1], x[0], x[1], x[2], x[3], bq[2], bq[3]);
              if (WIDE && s > 0) {
#pragma unroll
                for (int e = 0; e < 4; ++e) { r[m][0][e] = r[m][0][e] * 0.0078125f; r[m][1][e] = r[m][1][e] * 0.0078125f; }
              }
            }
          }
#pragma unroll
          for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              acc[m][2 * n2][e] = acc[m][2 * n2][e] + r[m][0][e];
              acc[m][2 * n2 + 1][e] = acc[m][2 * n2 + 1][e] + r[m][1][e];
            }
        }
      }
    }
    bool met = least < (kTiny << 1) - 1u;
    if (!WIDE)   // NaN: perhaps an infinite X against a zero term
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) met = met || isnan(acc[m][n][e]);
    return met;
  };
  if (__syncthreads_or(walk(std::false_type{}))) walk(std::true_type{});
  float* o = part + (size_t)blockIdx.x * BLK_SZ;
  const int g = ln >> 2, q = ln & 3;
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int n = 0; n < 4; ++n)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<float2*>(&o[(tap * C + m * 16 + g + 8 * h) * C + n * 8 + 2 * q]) =
            make_float2(acc[m][n][2 * h], acc[m][n][2 * h + 1]);
  // the bias: the staging threads' sums, in the threads' order
  __syncthreads();
  float* sS = reinterpret_cast<float*>(&sD[0][0]);   // [GT / 8][32]
  static_assert(GT / 8 * 32 * sizeof(float) <= sizeof(sD), "room for the sums");
  *reinterpret_cast<float4*>(&sS[threadIdx.x / (C / 4) * C + c4]) = sum;
  __syncthreads();
  if (threadIdx.x < C) {
    float v = sS[threadIdx.x];
    for (int r = 1; r < GT / 8; ++r) v = v + sS[r * C + threadIdx.x];
    o[9 * C * C + threadIdx.x] = v;
  }
}

// The stem's and the head's, FP32: a tile's X and DY are staged in shared memory, and a thread walks
// pixels with the 3 x 3 window of X in registers, so a pixel costs three loads of X for all taps.
//    4 -> 32  lane = co, four ci a thread (one 16-byte load of X): 36 sums
//   32 -> 1   lane = ci: 9 sums
// A warp takes half a row of a tile; the warps' sums are added at the end in a fixed order.  The next
// tile's values are fetched into registers behind the tile's arithmetic.  32 x 64 x 64 pixels, per call,
// with one load of X per multiply-add and no FMA -> this: 57 -> 16 and 63 -> 11 us (8 x 16 pixel tiles
// without the fetch ahead: 29, 44).
constexpr int WGW = 8;                     // warps of a weight-gradient block
template <int CIN, int COUT, typename XT>
__global__ void __launch_bounds__(32 * WGW, 2) k_wgrad(const XT* __restrict__ X, const float* __restrict__ DY, int B,
                                                       int H, int W, float* __restrict__ part) {
  constexpr bool STEM = CIN == 4 && COUT == 32;
  static_assert(STEM || (CIN == 32 && COUT == 1), "layer shape");
  static_assert(WGW == 2 * GH, "half a row a warp");
  constexpr int NTH = 32 * WGW;
  constexpr int R = 9 * CIN, NOUT = R * COUT + COUT;
  constexpr int NX = STEM ? 4 : 1;           // channels of a window pixel in a thread
  constexpr int NA = 9 * NX + 1;             // sums of a thread
  constexpr int XV = STEM ? 1 : 8, NXL = (GHP * CIN / XV + NTH - 1) / NTH;     // loads of X a thread, values each
  constexpr int DV = STEM ? 4 : 1, NDL = (GP * COUT / DV + NTH - 1) / NTH;     // of DY
  __shared__ __align__(16) float sX[GHP * CIN];
  __shared__ __align__(16) float sD[GP * COUT];
  __shared__ float sA[WGW][NA * 32];
  const int ln = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int nj = (W + TW - 1) / TW, ni = (H + GH - 1) / GH, ntiles = B * ni * nj;
  float acc[9][NX], accb = 0.f;
#pragma unroll
  for (int t = 0; t < 9; ++t)
#pragma unroll
    for (int q = 0; q < NX; ++q) acc[t][q] = 0.f;
  uint4 rx[STEM ? 1 : NXL];
  float rxf[STEM ? NXL : 1];
  float4 rd[STEM ? NDL : 1];
  float rdf = 0.f;
  auto fetch = [&](int tile) {   // a tile's X (zero outside the image) and DY to registers
    const int b = tile / (ni * nj), rem = tile - b * (ni * nj), i0 = rem / nj * GH, j0 = rem % nj * TW;
#pragma unroll
    for (int k = 0; k < NXL; ++k) {
      const int r = threadIdx.x + k * NTH, pix = r / (CIN / XV), c = r % (CIN / XV) * XV;
      const int gi = i0 + pix / WT - 1, gj = j0 + pix % WT - 1;
      const bool in = pix < GHP && gi >= 0 && gi < H && gj >= 0 && gj < W;
      const size_t o = (((size_t)b * H + gi) * W + gj) * CIN + c;
      if constexpr (STEM) {
        rxf[k] = in ? bfr(X[o]) : 0.f;
      } else {
        rx[k] = make_uint4(0u, 0u, 0u, 0u);
        if (in) rx[k] = *reinterpret_cast<const uint4*>(X + o);
      }
    }
#pragma unroll
    for (int k = 0; k < NDL; ++k) {
      const int r = threadIdx.x + k * NTH, pix = r / (COUT / DV), c = r % (COUT / DV) * DV;
      const int gi = i0 + pix / TW, gj = j0 + pix % TW;
      const bool in = pix < GP && gi < H && gj < W;
      const size_t o = (((size_t)b * H + gi) * W + gj) * COUT + c;
      if constexpr (STEM) {
        rd[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (in) rd[k] = *reinterpret_cast<const float4*>(DY + o);
      } else {
        rdf = in ? DY[o] : 0.f;
      }
    }
  };
  if ((int)blockIdx.x < ntiles) fetch(blockIdx.x);
  for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NXL; ++k) {
      const int r = threadIdx.x + k * NTH;
      if (r * XV < GHP * CIN) {
        if constexpr (STEM) {
          sX[r] = rxf[k];
        } else {
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&rx[k]);
          const float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
          const float2 c = __bfloat1622float2(h[2]), d = __bfloat1622float2(h[3]);
          *reinterpret_cast<float4*>(&sX[r * 8]) = make_float4(a.x, a.y, b.x, b.y);
          *reinterpret_cast<float4*>(&sX[r * 8 + 4]) = make_float4(c.x, c.y, d.x, d.y);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < NDL; ++k) {
      const int r = threadIdx.x + k * NTH;
      if (r * DV < GP * COUT) {
        if constexpr (STEM) *reinterpret_cast<float4*>(&sD[r * 4]) = rd[k];
        else sD[r] = rdf;
      }
    }
    __syncthreads();
    if (tile + (int)gridDim.x < ntiles) fetch(tile + gridDim.x);   // lands behind this tile's arithmetic
    const int ti = wp >> 1, t0 = (wp & 1) * (TW / 2);
    float x[3][3][NX];   // the 3 x 3 window of X
    auto column = [&](int c, int tj) {   // window column c from image column tj - 1
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const int o = ((ti + i) * WT + tj) * CIN;
        if constexpr (STEM) {
          const float4 v = *reinterpret_cast<const float4*>(&sX[o]);
          x[i][c][0] = v.x; x[i][c][1] = v.y; x[i][c][2] = v.z; x[i][c][3] = v.w;
        } else {
          x[i][c][0] = sX[o + ln];
        }
      }
    };
    column(0, t0);
    column(1, t0 + 1);
#pragma unroll 4
    for (int tj = t0; tj < t0 + TW / 2; ++tj) {
      column(2, tj + 2);
      const float d = sD[(ti * TW + tj) * COUT + (STEM ? ln : 0)];
      accb = accb + d;
#pragma unroll
      for (int t = 0; t < 9; ++t)
#pragma unroll
        for (int q = 0; q < NX; ++q) acc[t][q] = fmaf(x[t / 3][t % 3][q], d, acc[t][q]);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int q = 0; q < NX; ++q) { x[i][0][q] = x[i][1][q]; x[i][1][q] = x[i][2][q]; }
    }
  }
  float* o = part + (size_t)blockIdx.x * NOUT;
#pragma unroll
  for (int m = 0; m < NA; ++m) sA[wp][m * 32 + ln] = m < 9 * NX ? acc[m / NX % 9][m % NX] : accb;
  __syncthreads();
  for (int r = threadIdx.x; r < NA * 32; r += NTH) {
    const int m = r >> 5, l = r & 31;
    float v = sA[0][r];
    for (int w = 1; w < WGW; ++w) v = v + sA[w][r];
    if (m < 9 * NX) o[STEM ? m * COUT + l : m * CIN + l] = v;   // m = tap (x 4 + ci)
    else if (STEM || l == 0) o[R * COUT + l] = v;
  }
}

// grad[off + o] = sum_blk part[blk][o] (fixed order: WR threads of an output each take every WR-th block,
// then their sums in order); the weight part [9][CIN][COUT] first, then the COUT bias entries.  One
// thread per output left three SMs in four idle (21 us for the 9248 outputs of a block, 8.5 so; 32 threads an output 7.7,
// but a larger rounding error).
constexpr int WR = 8;
__global__ void __launch_bounds__(32 * WR) k_wgrad_reduce(const float* __restrict__ part, int nblk, int nout,
                                                          float* __restrict__ grad) {
  __shared__ float sh[WR][32];
  const int o = blockIdx.x * 32 + threadIdx.x;
  float s = 0.f;
  if (o < nout) {
#pragma unroll 10
    for (int b = threadIdx.y; b < nblk; b += WR) s = s + part[(size_t)b * nout + o];
  }
  sh[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y != 0 || o >= nout) return;
  for (int w = 1; w < WR; ++w) s = s + sh[w][threadIdx.x];
  grad[o] = s;
}

// ------------------------------------------------------------------ loss and optimiser
__global__ void k_loss_part(const float* __restrict__ out, const float* __restrict__ t, const float* __restrict__ mask,
                            int n, float* __restrict__ part) {
  __shared__ float s1[256], s2[256];
  float a = 0.f, m = 0.f;
  for (int i = blockIdx.x * 256 + threadIdx.x; i < n; i += gridDim.x * 256) {
    if (mask[i] > 0.f) {
      const float d = out[i] - t[i];
      a = a + d * d;
      m = m + 1.f;
    }
  }
  s1[threadIdx.x] = a;
  s2[threadIdx.x] = m;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) { s1[threadIdx.x] += s1[threadIdx.x + o]; s2[threadIdx.x] += s2[threadIdx.x + o]; }
    __syncthreads();
  }
  if (threadIdx.x == 0) { part[2 * blockIdx.x] = s1[0]; part[2 * blockIdx.x + 1] = s2[0]; }
}

constexpr int LOSS_BLOCKS = 148;   // blocks of k_loss_part
__global__ void k_loss_final(const float* __restrict__ part, int nblk, float* __restrict__ loss) {
  // staged by all threads (the loop's loads would each wait for memory), added in order by one
  __shared__ float sp[2 * LOSS_BLOCKS];
  for (int b = threadIdx.x; b < 2 * nblk; b += blockDim.x) sp[b] = part[b];
  __syncthreads();
  if (threadIdx.x != 0) return;
  float a = 0.f, m = 0.f;
  for (int b = 0; b < nblk; ++b) { a = a + sp[2 * b]; m = m + sp[2 * b + 1]; }
  loss[0] = m > 0.f ? a / m : 0.f;
  loss[1] = m;
}

__global__ void k_loss_grad(const float* __restrict__ out, const float* __restrict__ t, const float* __restrict__ mask,
                            int n, const float* __restrict__ loss, float* __restrict__ gout) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float m = loss[1];
  gout[i] = (mask[i] > 0.f && m > 0.f) ? 2.f * (out[i] - t[i]) / m : 0.f;
}

__global__ void k_adam(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       int n, float lr, float b1, float b2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  p[i] = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

// ------------------------------------------------------------------ solver-side kernels
// r0 = qq - A sp for every wet column (SolverSparse's matrix: diagonal rr, off-diagonals -sx_W,
// -sy_S, -sy, -sx) and block partial sums of r0^2.
__global__ void k_feat_resid(Dev d, double* __restrict__ r0, double* __restrict__ part) {
  __shared__ double sh[256];
  const int l = blockIdx.x * blockDim.x + threadIdx.x + 1;
  double v = 0.0;
  if (l <= d.g.lm) {
    const int lE = NB(d.g.lEC, l), lW = NB(d.g.lWC, l), lN = NB(d.g.lNC, l), lS = NB(d.g.lSC, l);
    const double* sp = d.s.sp;
    const double ax = d.s.rr[l - 1] * sp[l - 1] - d.s.sx[lW - 1] * sp[lW - 1] - d.s.sy[lS - 1] * sp[lS - 1] -
                      d.s.sy[l - 1] * sp[lN - 1] - d.s.sx[l - 1] * sp[lE - 1];
    const double r = d.s.qq[l - 1] - ax;
    r0[l - 1] = r;
    v = r * r;
  }
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

// One block of 256 threads: strided partial sums, then a tree in shared memory (fixed order).
__global__ void k_feat_sigma(const double* __restrict__ part, int nblk, int lm, double* __restrict__ sigma) {
  __shared__ double sh[256];
  double s = 0.0;
  for (int b = threadIdx.x; b < nblk; b += 256) s += part[b];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) sigma[0] = lm > 0 ? sqrt(sh[0] / lm) : 0.0;
}

__global__ void k_feat_write(Dev d, const int* __restrict__ pix, const double* __restrict__ r0,
                             const double* __restrict__ sigma, float* __restrict__ feat) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (l > d.g.lm) return;
  const double s = sigma[0];
  const double inv = s > 0.0 ? 1.0 / s : 0.0;
  float4 f;
  f.x = (float)(r0[l - 1] * inv);
  f.y = (float)((d.s.sp[l - 1] - d.s.spp[l - 1]) * inv);
  f.z = (float)(d.g.hhs[l - 1] / 30.0);
  f.w = 1.f;
  *reinterpret_cast<float4*>(feat + (size_t)pix[l - 1] * 4) = f;
}

__global__ void k_feat_scatter(int lm, const int* __restrict__ pix, const float* __restrict__ out,
                               const double* __restrict__ sigma, double* __restrict__ dz) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (l > lm) return;
  const double s = sigma[0];
  dz[l - 1] = s > 0.0 ? s * (double)out[pix[l - 1]] : 0.0;
}

__global__ void k_record(Dev d, const int* __restrict__ pix, const float* __restrict__ feat,
                         const double* __restrict__ sigma, float* __restrict__ rec) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (l > d.g.lm) return;
  const size_t p = (size_t)pix[l - 1];
  const float4 f = *reinterpret_cast<const float4*>(feat + p * 4);
  const double s = sigma[0];
  float* o = rec + p * 5;
  o[0] = f.x; o[1] = f.y; o[2] = f.z; o[3] = f.w;
  o[4] = s > 0.0 ? (float)((d.s.s[l - 1] - d.s.sp[l - 1]) / s) : 0.f;
}

dim3 tiles(int B, int H, int W) { return dim3((W + TW - 1) / TW, (H + TH - 1) / TH, B); }

}  // namespace

// ---------------------------------------------------------------------------- host side
size_t Workspace::bytes(int B, int H, int W, bool training) {
  const size_t P = (size_t)B * H * W;
  size_t s = 0;
  auto add = [&](size_t n) { s += (n + 255) / 256 * 256; };
  add(2 * SI3D_NET_BLOCKS * 9 * C * C * sizeof(bf16));   // wfwd, wbwd
  add((9 * 4 * C + C) * sizeof(float));
  add((9 * C + 1) * sizeof(float));
  const int nx = training ? SI3D_NET_BLOCKS + 1 : 2;
  for (int i = 0; i < nx; ++i) add(P * C * sizeof(bf16));
  if (training) {
    for (int i = 0; i < SI3D_NET_BLOCKS + 1; ++i) add(P * C * sizeof(float));   // y0..y4
    for (int i = 0; i < 2; ++i) add(P * C * sizeof(float));                     // G, DY
    for (int i = 0; i < 2; ++i) add(P * C * sizeof(bf16));                      // DYb of two layers
    add((size_t)WG_BLOCKS * (9 * C * C + C) * sizeof(float));                    // weight-gradient partials
  }
  return s;
}

bool Workspace::carve(void* base, size_t avail, int B, int H, int W, bool training) {
  if (!base || avail < bytes(B, H, W, training)) return false;
  const size_t P = (size_t)B * H * W;
  char* q = static_cast<char*>(base);
  auto take = [&](size_t n) { void* r = q; q += (n + 255) / 256 * 256; return r; };
  wfwd = static_cast<bf16*>(take(SI3D_NET_BLOCKS * 9 * C * C * sizeof(bf16) * 2));
  wbwd = wfwd + SI3D_NET_BLOCKS * 9 * C * C;
  stem = static_cast<float*>(take((9 * 4 * C + C) * sizeof(float)));
  head = static_cast<float*>(take((9 * C + 1) * sizeof(float)));
  const int nx = training ? SI3D_NET_BLOCKS + 1 : 2;
  for (int i = 0; i < SI3D_NET_BLOCKS + 1; ++i) x[i] = nullptr;
  for (int i = 0; i < nx; ++i) x[i] = static_cast<bf16*>(take(P * C * sizeof(bf16)));
  for (int i = 0; i < SI3D_NET_BLOCKS + 1; ++i) y[i] = nullptr;
  G = DY = nullptr;
  DYb[0] = DYb[1] = nullptr;
  part = nullptr;
  if (training) {
    for (int i = 0; i < SI3D_NET_BLOCKS + 1; ++i) y[i] = static_cast<float*>(take(P * C * sizeof(float)));
    G = static_cast<float*>(take(P * C * sizeof(float)));
    DY = static_cast<float*>(take(P * C * sizeof(float)));
    for (int i = 0; i < 2; ++i) DYb[i] = static_cast<bf16*>(take(P * C * sizeof(bf16)));
    part = static_cast<float*>(take((size_t)WG_BLOCKS * (9 * C * C + C) * sizeof(float)));
  }
  this->training = training;
  return true;
}

void prepare(const Workspace& ws, const float* params, cudaStream_t st) {
  const int n = SI3D_NET_BLOCKS * 9 * C * C;
  k_prep<<<(n + 255) / 256, 256, 0, st>>>(params, ws.wfwd, ws.wbwd, ws.stem, ws.head);
}

// Persistent grid of the convolution: every resident block of the device, at most one per tile.
int conv_bwd_blocks(int B, int H, int W) {
  int dev = 0, sms = 1, occ = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_conv32_bwd, 128, 0);
  const long long ntiles = (long long)B * ((H + TH - 1) / TH) * ((W + TW - 1) / TW);
  return (int)std::max(1LL, std::min(ntiles, (long long)sms * std::max(occ, 1)));
}

// Persistent grid of the tcgen05 convolution: one block per SM (its shared memory takes most of
// one), enabled once per device.
int conv_tc_blocks(int B, int H, int W) {
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  static bool attr_set[64] = {false};
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    cudaFuncSetAttribute(k_conv32_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM);
    attr_set[dev] = true;
  }
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long ntiles = (long long)B * ((H + TC_R - 1) / TC_R) * ((W + TC_W - 1) / TC_W);
  return (int)std::max(1LL, std::min(ntiles, (long long)sms));
}

// cuTensorMapEncodeTiled from the driver, looked up once.
PFN_cuTensorMapEncodeTiled_v12000 encode_tiled() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

// TMA map of a channels-last activation image [B][H][W][C] (bf16): boxes of 8 channels (16 bytes,
// the innermost extent) x 130 pixels x (TC_R + 2) rows of one image; coordinates outside the image
// read as zero.
bool activation_map(CUtensorMap* m, const bf16* x, int B, int H, int W) {
  PFN_cuTensorMapEncodeTiled_v12000 enc = encode_tiled();
  if (!enc || (reinterpret_cast<uintptr_t>(x) & 15u) != 0) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)B};
  const cuuint64_t strides[3] = {(cuuint64_t)C * sizeof(bf16), (cuuint64_t)W * C * sizeof(bf16),
                                 (cuuint64_t)H * W * C * sizeof(bf16)};
  const cuuint32_t box[4] = {8, (cuuint32_t)TC_WT, (cuuint32_t)(TC_R + 2), 1};
  const cuuint32_t elem[4] = {1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(x), dims, strides, box, elem,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int forward(const Workspace& ws, const float* params, const float* feat, int B, int H, int W, float* out,
            cudaStream_t st) {
  const float* bias0 = params + OFF_BLK + 9 * C * C;
  const dim3 grid((W + ST_W - 1) / ST_W, (H + TH - 1) / TH, B);
  CUtensorMap maps[SI3D_NET_BLOCKS];
  for (int k = 0; k < SI3D_NET_BLOCKS; ++k)
    if (!activation_map(&maps[k], ws.training ? ws.x[k] : ws.x[k & 1], B, H, W)) return SI3D_ECUDA;
  k_stem<<<grid, 32 * TH, 0, st>>>(feat, ws.stem, H, W, ws.x[0], ws.training ? ws.y[0] : nullptr);
  const int nb = conv_tc_blocks(B, H, W);
  for (int k = 0; k < SI3D_NET_BLOCKS; ++k) {
    bf16* xout = ws.training ? ws.x[k + 1] : ws.x[(k + 1) & 1];
    k_conv32_tc<<<nb, TC_THREADS, TC_SMEM, st>>>(maps[k], ws.wfwd + (size_t)k * 9 * C * C,
                                                  bias0 + (size_t)k * BLK_SZ, B, H, W, xout,
                                                  ws.training ? ws.y[k + 1] : nullptr);
  }
  const bf16* xl = ws.training ? ws.x[SI3D_NET_BLOCKS] : ws.x[SI3D_NET_BLOCKS & 1];
  k_head<<<grid, HD_T, 0, st>>>(xl, ws.head, H, W, out);
  return 0;
}

void backward(const Workspace& ws, const float* feat, const float* gout, int B, int H, int W, float* grad,
              cudaStream_t st) {
  const dim3 grid = tiles(B, H, W);
  // head
  k_wgrad<C, 1, bf16><<<WG_BLOCKS, 32 * WGW, 0, st>>>(ws.x[SI3D_NET_BLOCKS], gout, B, H, W, ws.part);
  k_wgrad_reduce<<<(9 * C + 1 + 31) / 32, dim3(32, WR), 0, st>>>(ws.part, WG_BLOCKS, 9 * C + 1, grad + OFF_HEAD_W);
  k_head_bwd<<<grid, TP, 0, st>>>(gout, ws.head, H, W, ws.y[SI3D_NET_BLOCKS], ws.G, ws.DY, ws.DYb[0]);
  const int nb = conv_bwd_blocks(B, H, W);
  for (int k = SI3D_NET_BLOCKS - 1, cur = 0; k >= 0; --k, cur ^= 1) {
    k_wgrad32<<<WG_BLOCKS, GT, 0, st>>>(ws.x[k], ws.DY, B, H, W, ws.part);
    k_wgrad_reduce<<<(BLK_SZ + 31) / 32, dim3(32, WR), 0, st>>>(ws.part, WG_BLOCKS, BLK_SZ, grad + OFF_BLK + k * BLK_SZ);
    k_conv32_bwd<<<nb, 128, 0, st>>>(ws.DYb[cur], ws.wbwd + (size_t)k * 9 * C * C, B, H, W, ws.G, ws.y[k], ws.DY,
                                     k > 0 ? ws.DYb[cur ^ 1] : nullptr);
  }
  k_wgrad<4, C, float><<<WG_BLOCKS, 32 * WGW, 0, st>>>(feat, ws.DY, B, H, W, ws.part);
  k_wgrad_reduce<<<(9 * 4 * C + C + 31) / 32, dim3(32, WR), 0, st>>>(ws.part, WG_BLOCKS, 9 * 4 * C + C, grad);
}

void features(const Dev& d, const int* pix, double* r0, double* part, double* sigma, float* feat, cudaStream_t st) {
  const int nb = (d.g.lm + 255) / 256;
  k_feat_resid<<<nb, 256, 0, st>>>(d, r0, part);
  k_feat_sigma<<<1, 256, 0, st>>>(part, nb, d.g.lm, sigma);
  k_feat_write<<<nb, 256, 0, st>>>(d, pix, r0, sigma, feat);
}

void scatter(int lm, const int* pix, const float* out, const double* sigma, double* dz, cudaStream_t st) {
  k_feat_scatter<<<(lm + 255) / 256, 256, 0, st>>>(lm, pix, out, sigma, dz);
}

void record(const Dev& d, const int* pix, const float* feat, const double* sigma, float* rec, cudaStream_t st) {
  k_record<<<(d.g.lm + 255) / 256, 256, 0, st>>>(d, pix, feat, sigma, rec);
}

int feature_partials(int lm) { return (lm + 255) / 256; }

}  // namespace learn
}  // namespace si3d

// ---------------------------------------------------------------------------- C ABI (training)
using si3d::learn::Workspace;

extern "C" {

size_t si3d_net_workspace_bytes(int B, int H, int W) {
  if (B < 1 || H < 1 || W < 1) return 0;
  return Workspace::bytes(B, H, W, true);
}

int si3d_net_forward(const float* params, const float* feat, int B, int H, int W, float* out, void* ws_ptr,
                     size_t ws_bytes) {
  if (!params || !feat || !out || B < 1 || H < 1 || W < 1) return SI3D_EDIMS;
  Workspace ws;
  if (!ws.carve(ws_ptr, ws_bytes, B, H, W, true)) return SI3D_EDIMS;
  si3d::learn::prepare(ws, params, 0);
  if (int rc = si3d::learn::forward(ws, params, feat, B, H, W, out, 0)) return rc;
  return cudaGetLastError() == cudaSuccess ? SI3D_OK : SI3D_ECUDA;
}

int si3d_net_loss(const float* out, const float* target, const float* mask, int n, float* gout, float* loss_dev) {
  if (!out || !target || !mask || !gout || !loss_dev || n < 1) return SI3D_EDIMS;
  constexpr int NB = si3d::learn::LOSS_BLOCKS;
  float* part = loss_dev + 2;   // the caller's loss buffer holds 2 + 2 * 148 floats
  si3d::learn::k_loss_part<<<NB, 256>>>(out, target, mask, n, part);
  si3d::learn::k_loss_final<<<1, 256>>>(part, NB, loss_dev);
  si3d::learn::k_loss_grad<<<(n + 255) / 256, 256>>>(out, target, mask, n, loss_dev, gout);
  return cudaGetLastError() == cudaSuccess ? SI3D_OK : SI3D_ECUDA;
}

int si3d_net_backward(const float* params, const float* feat, const float* gout, int B, int H, int W, float* grad,
                      void* ws_ptr, size_t ws_bytes) {
  if (!params || !feat || !gout || !grad || B < 1 || H < 1 || W < 1) return SI3D_EDIMS;
  Workspace ws;
  if (!ws.carve(ws_ptr, ws_bytes, B, H, W, true)) return SI3D_EDIMS;
  si3d::learn::backward(ws, feat, gout, B, H, W, grad, 0);
  return cudaGetLastError() == cudaSuccess ? SI3D_OK : SI3D_ECUDA;
}

int si3d_net_adam(float* params, const float* grad, float* m, float* v, int n, float lr, float beta1, float beta2,
                  float eps, int t) {
  if (!params || !grad || !m || !v || n < 1 || t < 1) return SI3D_EDIMS;
  const float c1 = 1.f - powf(beta1, (float)t), c2 = 1.f - powf(beta2, (float)t);
  si3d::learn::k_adam<<<(n + 255) / 256, 256>>>(params, grad, m, v, n, lr, beta1, beta2, eps, c1, c2);
  return cudaGetLastError() == cudaSuccess ? SI3D_OK : SI3D_ECUDA;
}

int si3d_net_sync(void) { return cudaDeviceSynchronize() == cudaSuccess ? SI3D_OK : SI3D_ECUDA; }

}  // extern "C"
