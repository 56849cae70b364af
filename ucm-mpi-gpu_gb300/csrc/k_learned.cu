// k_learned.cu -- the learned warm start's network: forward, loss and
// backward kernels, BF16 operands on the tensor cores (mma.sync m16n8k16)
// with FP32 accumulation, and Adam.
//
// Tensors are per level, channel-innermost ([pixel][channel]), the patches of
// a batch back to back (LnPatch offsets).  Activations are BF16; gradients
// are FP32 and are rounded to BF16 only where a convolution feeds them to the
// tensor cores.
//
//   k_ln_conv    3 x 3 convolution as an implicit GEMM over an 8 x 16 output
//                tile: the tile's input with a 1-pixel halo and the weights
//                of a chunk of output channels are staged in shared memory;
//                each of 4 warps computes two 16-pixel rows x the chunk.
//                Forward (ReLU to BF16, or the head to FP32), and the
//                data gradient (the masked FP32 output gradient staged as
//                BF16, convolved with the flipped, transposed weights).
//   k_ln_wgrad   weight and bias gradients: a CTA accumulates dW = dZ^T X of
//                all taps over its share of the tiles on the tensor cores,
//                then adds it to the FP32 gradient.
//   pooling, the gradients of pooling, up-sampling and concatenation, the subspace
//   loss reductions and its gradient, Adam, the weights' BF16 copies.
#include <cuda_bf16.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "k_block.h"
#include "k_learned.h"
#include "per_device.h"

namespace gpb {

const LnConv kLnNet[kLnConvs] = {
    {16, 16, 1},  {16, 16, 1},  {16, 32, 1}, {32, 32, 1}, {32, 64, 1}, {64, 64, 1}, {64, 64, 1}, {64, 64, 1},
    {128, 64, 1}, {64, 64, 1},  {96, 32, 1}, {32, 32, 1}, {48, 16, 1}, {16, 16, 1}, {16, 32, 0}};

static void conv_offsets(size_t* wo, size_t* bo, size_t* total) {
  size_t o = 0;
  for (int i = 0; i < kLnConvs; i++) {
    wo[i] = o;
    o += (size_t)kLnNet[i].cout * 9 * kLnNet[i].cin;
    bo[i] = o;
    o += kLnNet[i].cout;
  }
  *total = o;
}

size_t ln_nparams() {
  size_t wo[kLnConvs], bo[kLnConvs], t;
  conv_offsets(wo, bo, &t);
  return t;
}

namespace {

typedef __nv_bfloat16 bf16;
constexpr int TH = 8, TW = 16, HP = TH + 2, WP = TW + 2, NHALO = HP * WP;  // tile, halo tile
constexpr int kConvThreads = 128;

__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *(const uint32_t*)&v;
}

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

// A convolution's BF16 input, CIN channels of pixel (y, x) of a patch: with
// C1 = 0 one tensor; with C1 > 0 the concatenation of an up-sampled coarser
// tensor (C1 channels, nearest) and a skip tensor, read where they lie.
struct LnIn {
  const bf16* x;        // the tensor, or the skip tensor
  const bf16* coarse;   // C1 channels at the next coarser level
  const LnPatch* cp;    // that level's patches
};
template <int CIN, int C1>
__device__ __forceinline__ uint4 ln_in8(const LnIn& in, const LnPatch& P, const LnPatch& Q, int y, int x, int c) {
  if (C1 > 0 && c < C1)
    return *(const uint4*)(in.coarse + (Q.off + (long long)(y >> 1) * Q.W + (x >> 1)) * C1 + c);
  return *(const uint4*)(in.x + (P.off + (long long)y * P.W + x) * (CIN - C1) + c - C1);
}

// MODE 0: forward, ReLU, BF16 out.  1: forward head, FP32 out.
// 2: data gradient: dA is the FP32 output gradient of the layer being
//    differentiated (CIN = its channels), masked by its BF16 activation
//    (mask, may be null) and rounded to BF16; w is the flipped, transposed
//    weight; FP32 out, no bias.
// A persistent CTA stages its weights once and walks the tiles blockIdx.x,
// + gridDim.x, ...; fragments come by ldmatrix, one instruction for the four
// registers that plain loads took four for.  Bound by the staging (memory)
// for the thin layers, by fragment loads and mma.sync for the wide ones.
// Measured, forward of 617 kpx, all 15: 357 us, from 392 us with the weights
// staged per tile and 4-byte fragment loads.
template <int CIN, int CO, int MODE, int C1>
__global__ void __launch_bounds__(kConvThreads) k_ln_conv(const LnPatch* __restrict__ lp,
                                                          const LnTile* __restrict__ tiles, int ntiles, LnIn in,
                                                          const float* __restrict__ dA,
                                                          const bf16* __restrict__ mask,
                                                          const bf16* __restrict__ w, const float* __restrict__ bias,
                                                          void* __restrict__ out, int cout_total) {
  constexpr int SI = CIN + 8, SW = 9 * CIN + 8;  // padded shared row strides (bank spread)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  bf16* in_s = (bf16*)smem_raw;
  bf16* w_s = in_s + NHALO * SI;
  const int co0 = blockIdx.y * CO;
  // this CTA's output channels of the weights
  for (int idx = threadIdx.x; idx < CO * (9 * CIN / 8); idx += blockDim.x) {
    const int r = idx / (9 * CIN / 8), q = idx % (9 * CIN / 8);
    *(uint4*)(w_s + r * SW + q * 8) = *(const uint4*)(w + (long long)(co0 + r) * 9 * CIN + q * 8);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3;
  float bs[CO / 8][2];
#pragma unroll
  for (int nt = 0; nt < CO / 8; nt++) {
    bs[nt][0] = MODE < 2 ? bias[co0 + nt * 8 + 2 * tg] : 0.f;
    bs[nt][1] = MODE < 2 ? bias[co0 + nt * 8 + 2 * tg + 1] : 0.f;
  }
  // ldmatrix rows: A: tile pixel (lane & 15) at channel half lane >> 4;
  // B: output channel (lane & 7) + 8 (lane >> 4) at channel half (lane >> 3) & 1
  const bf16* arow = in_s + (2 * warp * WP + (lane & 15)) * SI + 8 * (lane >> 4);
  const bf16* brow = w_s + ((lane & 7) + 8 * (lane >> 4)) * SW + 8 * ((lane >> 3) & 1);
  for (int ti = blockIdx.x; ti < ntiles; ti += gridDim.x) {
    const LnTile t = tiles[ti];
    const LnPatch P = lp[t.patch], Q = C1 > 0 ? in.cp[t.patch] : P;
    __syncthreads();
    // the input tile with its halo (zeros outside the patch)
    for (int idx = threadIdx.x; idx < NHALO * (CIN / 8); idx += blockDim.x) {
      const int h = idx / (CIN / 8), q = idx % (CIN / 8);
      const int y = t.y0 - 1 + h / WP, x = t.x0 - 1 + h % WP;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (y >= 0 && y < P.H && x >= 0 && x < P.W) {
        if constexpr (MODE == 2) {
          const long long pix = P.off + (long long)y * P.W + x;
          const float* gp = dA + pix * CIN + q * 8;
          const float4 g0 = *(const float4*)gp, g1 = *(const float4*)(gp + 4);
          float f[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
          if (mask) {
            const uint4 mk = *(const uint4*)(mask + pix * CIN + q * 8);
            const bf16* m = (const bf16*)&mk;
#pragma unroll
            for (int k = 0; k < 8; k++)
              if (!(__bfloat162float(m[k]) > 0.f)) f[k] = 0.f;
          }
          v = make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]), pack2(f[4], f[5]), pack2(f[6], f[7]));
        } else {
          v = ln_in8<CIN, C1>(in, P, Q, y, x, q * 8);
        }
      }
      *(uint4*)(in_s + h * SI + q * 8) = v;
    }
    __syncthreads();
    float acc[2][CO / 8][4];
#pragma unroll
    for (int mt = 0; mt < 2; mt++)
#pragma unroll
      for (int nt = 0; nt < CO / 8; nt++)
#pragma unroll
        for (int k = 0; k < 4; k++) acc[mt][nt][k] = 0.f;
#pragma unroll 1
    for (int tap = 0; tap < 9; tap++) {
      const bf16* at = arow + ((tap / 3) * WP + tap % 3) * SI;
      const bf16* bt = brow + tap * CIN;
#pragma unroll
      for (int kc = 0; kc < CIN / 16; kc++) {
        uint32_t a[2][4];
        ldsm4(a[0], at + kc * 16);
        ldsm4(a[1], at + WP * SI + kc * 16);
#pragma unroll
        for (int nt = 0; nt < CO / 8; nt += 2) {
          uint32_t b[4];
          ldsm4(b, bt + nt * 8 * SW + kc * 16);
#pragma unroll
          for (int mt = 0; mt < 2; mt++) {
            mma_bf16(acc[mt][nt], a[mt][0], a[mt][1], a[mt][2], a[mt][3], b[0], b[1]);
            mma_bf16(acc[mt][nt + 1], a[mt][0], a[mt][1], a[mt][2], a[mt][3], b[2], b[3]);
          }
        }
      }
    }
    // accumulator rows are tile pixels x = g (c0, c1) and g + 8 (c2, c3) of
    // tile row 2 warp + mt; columns are channels 2 tg, 2 tg + 1
#pragma unroll
    for (int mt = 0; mt < 2; mt++) {
      const int y = t.y0 + 2 * warp + mt;
      if (y >= P.H) continue;
#pragma unroll
      for (int half = 0; half < 2; half++) {
        const int x = t.x0 + g + 8 * half;
        if (x >= P.W) continue;
        const long long pix = P.off + (long long)y * P.W + x;
#pragma unroll
        for (int nt = 0; nt < CO / 8; nt++) {
          const int ch = co0 + nt * 8 + 2 * tg;
          float v0 = acc[mt][nt][2 * half], v1 = acc[mt][nt][2 * half + 1];
          if constexpr (MODE == 0) {
            v0 = fmaxf(v0 + bs[nt][0], 0.f);
            v1 = fmaxf(v1 + bs[nt][1], 0.f);
            *(uint32_t*)((bf16*)out + pix * cout_total + ch) = pack2(v0, v1);
          } else if constexpr (MODE == 1) {
            *(float2*)((float*)out + pix * cout_total + ch) = make_float2(v0 + bs[nt][0], v1 + bs[nt][1]);
          } else {
            *(float2*)((float*)out + pix * cout_total + ch) = make_float2(v0, v1);
          }
        }
      }
    }
  }
}

__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm2t(uint32_t (&r)[2], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1])
               : "r"((uint32_t)__cvta_generic_to_shared(p)));
}

// dW[n][tap][c] += sum over pixels of dZ[p][n] X[p + tap][c] for all nine
// taps and the CTA's CC input channels (from c0 = blockIdx.y * CC), over the
// tiles blockIdx.x, + gridDim.x, ...; db[n] += sum dZ[p][n] in the first
// chunk's CTAs.  dZ = BF16(dA * (mask > 0)).
// A GEMM over pixels, 16 (one tile row) per step: the tile's dZ and its X
// with the halo are staged once, pixel-major as they lie in memory, and
// ldmatrix.trans turns them into fragments, so a tap is only another row
// offset.  Warp (wc, wk) keeps the sums of CC / (8 WC) blocks of 8 input
// channels x 9 taps x COUT over the tile rows wk, wk + 8 / WC, ... in
// registers over all its tiles; the row groups are added in shared memory and
// leave with one atomic per weight and CTA.
// Bound by reading dA (FP32), mask and X for the thin layers and by the
// tensor pipe for 64 channels.  Measured for one gradient of 16 patches of
// 256^2, all 15 layers: 0.99 ms; a CTA per (tap, 16 channels), which
// staged every tile 9 CIN / 16 times and transposed it with 2-byte stores,
// took 4.24 ms.
template <int CIN, int CC, int COUT, int WC>
struct WgradCfg {
  static constexpr int WK = 8 / WC, CPW = CC / 8 / WC, NT = COUT / 16;
  static constexpr int ZP = COUT + 8, XP = CC + 8;  // row pitches: 16-byte rows in distinct banks
  static constexpr size_t stage = ((size_t)TH * TW * ZP + (size_t)NHALO * XP) * sizeof(bf16);
  static constexpr size_t sums = WK > 1 ? (size_t)COUT * 9 * CC * sizeof(float) : 0;
  static constexpr size_t smem = stage > sums ? stage : sums;
  static_assert(CPW * WC * 8 == CC && CIN % CC == 0, "channel split");
};
template <int CIN, int CC, int COUT, int WC, int C1>
__global__ void __launch_bounds__(256) k_ln_wgrad(const LnPatch* __restrict__ lp, const LnTile* __restrict__ tiles,
                                                  int ntiles, const float* __restrict__ dA,
                                                  const bf16* __restrict__ mask, LnIn X, float* __restrict__ dW,
                                                  float* __restrict__ db) {
  using G = WgradCfg<CIN, CC, COUT, WC>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  bf16* dz_s = (bf16*)smem_raw;            // [128][ZP]
  bf16* x_s = dz_s + TH * TW * G::ZP;      // [NHALO][XP]
  __shared__ float db_s[256];
  const int c0 = blockIdx.y * CC;
  const bool bias_cta = blockIdx.y == 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wc = warp % WC, wk = warp / WC;
  float acc[G::CPW][9][G::NT][4];
#pragma unroll
  for (int ct = 0; ct < G::CPW; ct++)
#pragma unroll
    for (int t = 0; t < 9; t++)
#pragma unroll
      for (int n = 0; n < G::NT; n++)
#pragma unroll
        for (int k = 0; k < 4; k++) acc[ct][t][n][k] = 0.f;
  float dbacc = 0.f;
  for (int ti = blockIdx.x; ti < ntiles; ti += gridDim.x) {
    const LnTile t = tiles[ti];
    const LnPatch P = lp[t.patch], Q = C1 > 0 ? X.cp[t.patch] : P;
    __syncthreads();
    for (int idx = threadIdx.x; idx < TH * TW * (COUT / 8); idx += blockDim.x) {
      const int px = idx / (COUT / 8), q = idx % (COUT / 8);
      const int y = t.y0 + px / TW, x = t.x0 + px % TW;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (y < P.H && x < P.W) {
        const long long pix = P.off + (long long)y * P.W + x;
        const float4 g0 = *(const float4*)(dA + pix * COUT + q * 8), g1 = *(const float4*)(dA + pix * COUT + q * 8 + 4);
        float f[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
        if (mask) {
          const uint4 mk = *(const uint4*)(mask + pix * COUT + q * 8);
          const bf16* m = (const bf16*)&mk;
#pragma unroll
          for (int k = 0; k < 8; k++)
            if (!(__bfloat162float(m[k]) > 0.f)) f[k] = 0.f;
        }
        v = make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]), pack2(f[4], f[5]), pack2(f[6], f[7]));
      }
      *(uint4*)(dz_s + px * G::ZP + q * 8) = v;
    }
    // zeros outside the patch; a pixel of the tile outside it has dZ = 0
    for (int idx = threadIdx.x; idx < NHALO * (CC / 8); idx += blockDim.x) {
      const int h = idx / (CC / 8), q = idx % (CC / 8);
      const int y = t.y0 - 1 + h / WP, x = t.x0 - 1 + h % WP;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (y >= 0 && y < P.H && x >= 0 && x < P.W)
        v = ln_in8<CIN, C1>(X, P, Q, y, x, c0 + q * 8);
      *(uint4*)(x_s + h * G::XP + q * 8) = v;
    }
    __syncthreads();
    if (bias_cta) {  // thread = channel + COUT * share of the pixels
      const int n = threadIdx.x % COUT, part = threadIdx.x / COUT;
      constexpr int PER = TH * TW * COUT / 256;
      float s = 0.f;
#pragma unroll 4
      for (int px = part * PER; px < (part + 1) * PER; px++) s += __bfloat162float(dz_s[px * G::ZP + n]);
      dbacc += s;
    }
#pragma unroll 1
    for (int row = wk; row < TH; row += G::WK) {
      uint32_t a[G::NT][4];
#pragma unroll
      for (int n = 0; n < G::NT; n++)
        ldsm4t(a[n], dz_s + (row * TW + (lane & 7) + ((lane >> 4) & 1) * 8) * G::ZP + n * 16 + ((lane >> 3) & 1) * 8);
#pragma unroll
      for (int tap = 0; tap < 9; tap++)
#pragma unroll
        for (int ct = 0; ct < G::CPW; ct++) {
          uint32_t b[2];
          ldsm2t(b, x_s + ((row + tap / 3) * WP + tap % 3 + (lane & 15)) * G::XP + (wc * G::CPW + ct) * 8);
#pragma unroll
          for (int n = 0; n < G::NT; n++) mma_bf16(acc[ct][tap][n], a[n][0], a[n][1], a[n][2], a[n][3], b[0], b[1]);
        }
    }
  }
  __syncthreads();
  const int g = lane >> 2, tg = lane & 3;
  float* sums = (float*)smem_raw;  // [COUT][9][CC]
  if constexpr (G::WK > 1) {
    for (int i = threadIdx.x; i < COUT * 9 * CC; i += blockDim.x) sums[i] = 0.f;
    __syncthreads();
  }
#pragma unroll
  for (int ct = 0; ct < G::CPW; ct++)
#pragma unroll
    for (int tap = 0; tap < 9; tap++)
#pragma unroll
      for (int n = 0; n < G::NT; n++)
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const int o = n * 16 + g + 8 * (k >> 1), c = (wc * G::CPW + ct) * 8 + 2 * tg + (k & 1);
          if constexpr (G::WK > 1)
            atomicAdd(sums + (o * 9 + tap) * CC + c, acc[ct][tap][n][k]);
          else
            atomicAdd(dW + ((long long)o * 9 + tap) * CIN + c0 + c, acc[ct][tap][n][k]);
        }
  if (bias_cta) db_s[threadIdx.x] = dbacc;
  __syncthreads();
  if constexpr (G::WK > 1) {
    for (int i = threadIdx.x; i < COUT * 9 * CC; i += blockDim.x)
      atomicAdd(dW + (long long)(i / CC) * CIN + c0 + i % CC, sums[i]);
  }
  if (bias_cta && threadIdx.x < COUT) {
    float s = 0.f;
    for (int i = threadIdx.x; i < 256; i += COUT) s += db_s[i];
    atomicAdd(db + threadIdx.x, s);
  }
}

// ---------------------------------------------------------- resampling
// 2 x 2 mean over the pixels that exist, BF16, C channels
__global__ void k_ln_pool(const LnPatch* __restrict__ lo, const LnPatch* __restrict__ hi, int npatch, int C,
                          const bf16* __restrict__ in, bf16* __restrict__ out) {
  const int p = blockIdx.y;
  const LnPatch S = lo[p], D = hi[p];  // source (fine), destination (coarse)
  const uint32_t nq = C / 8, total = (uint32_t)D.H * D.W * nq;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const uint32_t q = i % nq, px = i / nq;
    const int y = (int)(px / D.W), x = (int)(px % D.W);
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    int n = 0;
    for (int a = 0; a < 2; a++)
      for (int b = 0; b < 2; b++) {
        const int yy = 2 * y + a, xx = 2 * x + b;
        if (yy >= S.H || xx >= S.W) continue;
        const uint4 v = *(const uint4*)(in + (S.off + (long long)yy * S.W + xx) * C + q * 8);
        const bf16* e = (const bf16*)&v;
#pragma unroll
        for (int k = 0; k < 8; k++) s[k] += __bfloat162float(e[k]);
        n++;
      }
    const float r = 1.f / (float)n;
    *(uint4*)(out + (D.off + px) * C + q * 8) =
        make_uint4(pack2(s[0] * r, s[1] * r), pack2(s[2] * r, s[3] * r), pack2(s[4] * r, s[5] * r),
                   pack2(s[6] * r, s[7] * r));
  }
}

// The resampling gradients move 4 channels (16 bytes) per thread with 32-bit
// indices (a level of a patch has at most 2^26 pixels and 2^31 / 4 groups of
// channels); one channel per thread with 64-bit divisions took 300 us of
// one gradient of 16 patches of 256^2, against 153 us.
// dS[y][x] += dP[y/2][x/2] / count(y/2, x/2), FP32
__global__ void k_ln_pool_bwd(const LnPatch* __restrict__ lo, const LnPatch* __restrict__ hi, int C,
                              const float* __restrict__ dP, float* __restrict__ dS) {
  const int p = blockIdx.y;
  const LnPatch S = lo[p], D = hi[p];
  const uint32_t nq = C / 4, total = (uint32_t)S.H * S.W * nq;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const uint32_t q = i % nq, px = i / nq;
    const int y = (int)(px / S.W), x = (int)(px % S.W), cy = y >> 1, cx = x >> 1;
    const float n = (float)((min(2 * cy + 2, S.H) - 2 * cy) * (min(2 * cx + 2, S.W) - 2 * cx));
    float4* d = (float4*)(dS + (S.off + px) * C) + q;
    const float4 g = *((const float4*)(dP + (D.off + (long long)cy * D.W + cx) * C) + q);
    float4 v = *d;
    v.x += g.x / n;
    v.y += g.y / n;
    v.z += g.z / n;
    v.w += g.w / n;
    *d = v;
  }
}

// gradient of the concatenation [up(coarse), skip]: the coarse part summed over each 2 x 2 block, the
// skip part copied, FP32
__global__ void k_ln_upcat_bwd_coarse(const LnPatch* __restrict__ lo, const LnPatch* __restrict__ hi, int C1,
                                      int C2, const float* __restrict__ dC, float* __restrict__ dcoarse) {
  const int p = blockIdx.y;
  const LnPatch F = lo[p], Q = hi[p];
  const int C = C1 + C2;
  const uint32_t nq = C1 / 4, total = (uint32_t)Q.H * Q.W * nq;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const uint32_t q = i % nq, px = i / nq;
    const int y = (int)(px / Q.W), x = (int)(px % Q.W);
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int a = 0; a < 2; a++)
#pragma unroll
      for (int b = 0; b < 2; b++) {
        const int yy = 2 * y + a, xx = 2 * x + b;
        if (yy >= F.H || xx >= F.W) continue;
        const float4 v = *((const float4*)(dC + (F.off + (long long)yy * F.W + xx) * C) + q);
        s.x += v.x;
        s.y += v.y;
        s.z += v.z;
        s.w += v.w;
      }
    *((float4*)(dcoarse + (Q.off + px) * C1) + q) = s;
  }
}
__global__ void k_ln_upcat_bwd_skip(const LnPatch* __restrict__ lo, int C1, int C2, const float* __restrict__ dC,
                                    float* __restrict__ dskip) {
  const int p = blockIdx.y;
  const LnPatch F = lo[p];
  const int C = C1 + C2;
  const uint32_t nq = C2 / 4, total = (uint32_t)F.H * F.W * nq;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const uint32_t q = i % nq, px = i / nq;
    *((float4*)(dskip + (F.off + px) * C2) + q) = *((const float4*)(dC + (F.off + px) * C + C1) + q);
  }
}

// ------------------------------------------------------------ features
__global__ void k_ln_features(const LnPatch* __restrict__ lp, const float* __restrict__ mpb,
                              const float* __restrict__ deg, bf16* __restrict__ x) {
  const LnPatch P = lp[blockIdx.y];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (long long)P.H * P.W;
       i += (long long)gridDim.x * blockDim.x) {
    const long long q = P.off + i;
    uint4 v0 = make_uint4(pack2(mpb[q], deg[q] * (1.f / 81.f)), 0u, 0u, 0u);
    *(uint4*)(x + q * kLnIn) = v0;
    *(uint4*)(x + q * kLnIn + 8) = make_uint4(0u, 0u, 0u, 0u);
  }
}
__global__ void k_ln_features_from(const LnPatch* __restrict__ lp, const PatchDev* __restrict__ pd,
                                   const float* __restrict__ mpb, const float* __restrict__ deg,
                                   bf16* __restrict__ x) {
  const LnPatch P = lp[blockIdx.y];
  const PatchDev D = pd[blockIdx.y];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < (long long)P.H * P.W;
       i += (long long)gridDim.x * blockDim.x) {
    const long long q = P.off + i;
    *(uint4*)(x + q * kLnIn) = make_uint4(pack2(mpb[D.pix + i], deg[D.vec + i] * (1.f / 81.f)), 0u, 0u, 0u);
    *(uint4*)(x + q * kLnIn + 8) = make_uint4(0u, 0u, 0u, 0u);
  }
}

// ------------------------------------------------------------------ loss
// Rows of 4 consecutive pixels per warp pass through shared memory, so a
// pixel's 32 fields and 9 targets reach every lane as 16-byte broadcasts
// instead of 41 shuffles.
constexpr int kGramLen = kLnOut * kLnOut + kLnTargets * kLnOut;
constexpr int kVPitch = 12;
struct LnRows {
  float y[4][kLnOut];
  float v[4][kVPitch];
};
// a lane's share of 4 pixels q, q + step, .. (zeros from the n-th on), held in
// registers while the warp works on the previous 4
struct LnShare {
  float4 y;
  float v[2];
};
__device__ __forceinline__ LnShare ln_fetch(const float* __restrict__ y, const float* __restrict__ v, long long q,
                                            long long step, int n, int lane) {
  LnShare f;
  const int px = lane >> 3;
  f.y = px < n ? *(const float4*)(y + (q + px * step) * kLnOut + 4 * (lane & 7)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int i = lane + 32 * h, p = i / kLnTargets;
    f.v[h] = i < 4 * kLnTargets && p < n ? v[(q + p * step) * kLnTargets + i % kLnTargets] : 0.f;
  }
  return f;
}
__device__ __forceinline__ void ln_store(LnRows& r, const LnShare& f, int lane) {
  __syncwarp();
  *(float4*)&r.y[lane >> 3][4 * (lane & 7)] = f.y;
  r.v[lane / kLnTargets][lane % kLnTargets] = f.v[0];
  if (lane + 32 < 4 * kLnTargets) r.v[(lane + 32) / kLnTargets][(lane + 32) % kLnTargets] = f.v[1];
  __syncwarp();
}
__device__ __forceinline__ void ln_row(const LnRows& r, int p, float (&yk)[kLnOut], float (&vi)[kVPitch]) {
#pragma unroll
  for (int k = 0; k < kLnOut; k += 4) {
    const float4 f = *(const float4*)&r.y[p][k];
    yk[k] = f.x, yk[k + 1] = f.y, yk[k + 2] = f.z, yk[k + 3] = f.w;
  }
#pragma unroll
  for (int k = 0; k < kVPitch; k += 4) {
    const float4 f = *(const float4*)&r.v[p][k];
    vi[k] = f.x, vi[k + 1] = f.y, vi[k + 2] = f.z, vi[k + 3] = f.w;
  }
}

// per patch: G = Y^T Y (32 x 32) and B = V^T Y (9 x 32), FP64 sums of FP32
// per-warp partials; lane j owns column j.  The warps of a CTA are summed in
// shared memory before the atomics: 138 us for 16 patches of 256^2, from 358
// us with 5.5 M FP64 atomics and 41 shuffles per pixel.
__global__ void __launch_bounds__(256) k_ln_gram(const LnPatch* __restrict__ lp, const float* __restrict__ y,
                                                 const float* __restrict__ v, double* __restrict__ gb) {
  __shared__ __align__(16) LnRows rows[8];
  __shared__ float part[8][kGramLen];
  const LnPatch P = lp[blockIdx.y];
  const long long N = (long long)P.H * P.W;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long w0 = (long long)blockIdx.x * 8 + warp, nw = (long long)gridDim.x * 8;
  LnRows& r = rows[warp];
  if (lane < 4 * (kVPitch - kLnTargets)) r.v[lane / 3][kLnTargets + lane % 3] = 0.f;
  float G[kLnOut], B[kLnTargets];
#pragma unroll
  for (int k = 0; k < kLnOut; k++) G[k] = 0.f;
#pragma unroll
  for (int i = 0; i < kLnTargets; i++) B[i] = 0.f;
  auto count = [&](long long p) { return p < N ? (int)min((N - p + nw - 1) / nw, 4LL) : 0; };
  LnShare next = ln_fetch(y, v, P.off + w0, nw, count(w0), lane);
  for (long long p = w0; p < N; p += 4 * nw) {
    ln_store(r, next, lane);
    next = ln_fetch(y, v, P.off + p + 4 * nw, nw, count(p + 4 * nw), lane);
#pragma unroll
    for (int k4 = 0; k4 < 4; k4++) {
      float yk[kLnOut], vi[kVPitch];
      ln_row(r, k4, yk, vi);
      const float yj = r.y[k4][lane];
#pragma unroll
      for (int k = 0; k < kLnOut; k++) G[k] = fmaf(yj, yk[k], G[k]);
#pragma unroll
      for (int i = 0; i < kLnTargets; i++) B[i] = fmaf(vi[i], yj, B[i]);
    }
  }
#pragma unroll
  for (int k = 0; k < kLnOut; k++) part[warp][k * kLnOut + lane] = G[k];  // G is symmetric
#pragma unroll
  for (int i = 0; i < kLnTargets; i++) part[warp][kLnOut * kLnOut + i * kLnOut + lane] = B[i];
  __syncthreads();
  double* o = gb + (long long)blockIdx.y * kGramLen;
  for (int e = threadIdx.x; e < kGramLen; e += blockDim.x) {
    double s = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) s += (double)part[w][e];
    atomicAdd(o + e, s);
  }
}

// per patch, from G and B: C1 = B (G + eps I)^-1 (9 x 32) and C2 = C1^T C1
// (32 x 32) into cm, and the loss 9 - <C1, B>; bad is set where the
// regularised G is not positive definite.  One CTA per patch in FP64 with
// unfused operations in the order of a sequential Cholesky inverse, so the
// values are those of ln_solve_host.  Bound by the latency of the FP64 roots,
// quotients and subtraction chains: 147 us for any number of patches up to the
// SMs (few patches solve on the host, see kHostSolve).
__global__ void __launch_bounds__(256) k_ln_solve(const double* __restrict__ gb, float* __restrict__ cm,
                                                  double* __restrict__ loss, int* __restrict__ bad) {
  constexpr int K = kLnOut, T = kLnTargets, LP = K + 1;
  __shared__ double A[K * LP], Gi[K * LP], Bs[T * K], C1[T * K], red[T * K];
  const double* g = gb + (long long)blockIdx.x * kGramLen;
  const int tid = threadIdx.x, lane = tid & 31;
  double tr = 0;
  for (int i = 0; i < K; i++) tr = __dadd_rn(tr, g[i * K + i]);
  const double eps = __dadd_rn(__ddiv_rn(__dmul_rn(1e-4, tr), (double)K), 1e-30);
  for (int i = tid; i < K * K; i += 256) A[(i / K) * LP + i % K] = i / K == i % K ? __dadd_rn(g[i], eps) : g[i];
  for (int i = tid; i < T * K; i += 256) Bs[i] = g[K * K + i];
  __syncthreads();
  // Each element's products are subtracted in ascending k, as a dot product
  // would; the columns advance together.  A becomes L; Gi starts as I and
  // becomes L^-1, then (L L^T)^-1.
  __shared__ int fail;
  if (tid == 0) fail = 0;
  for (int e = tid; e < K * K; e += 256) Gi[(e / K) * LP + e % K] = e / K == e % K ? 1.0 : 0.0;
  __syncthreads();
  for (int j = 0; j < K; j++) {
    const double d = A[j * LP + j];
    if (tid == 0 && !(d > 0)) fail = 1;
    const double s = __dsqrt_rn(d > 0 ? d : 1.0);
    double l = 0;
    if (tid < 32) {
      if (lane > j) l = __ddiv_rn(A[lane * LP + j], s);
    } else if (tid < 64) {
      l = __ddiv_rn(Gi[j * LP + lane], s);  // row j of L^-1, column = lane
    }
    __syncthreads();
    if (tid < 32) {
      if (lane >= j) A[lane * LP + j] = lane == j ? s : l;
    } else if (tid < 64) {
      Gi[j * LP + lane] = l;
    }
    __syncthreads();
    for (int e = tid; e < K * K; e += 256) {
      const int r = e / K, q = e % K;
      if (r <= j) continue;
      const double lr = A[r * LP + j];
      if (q > j && q <= r) A[r * LP + q] = __dsub_rn(A[r * LP + q], __dmul_rn(lr, A[q * LP + j]));
      Gi[r * LP + q] = __dsub_rn(Gi[r * LP + q], __dmul_rn(lr, Gi[j * LP + q]));
    }
    __syncthreads();
  }
  if (tid < 32) {  // L^T x = z, lane = column
    for (int i = K - 1; i >= 0; i--) {
      double v = Gi[i * LP + lane];
#pragma unroll 8
      for (int k = i + 1; k < K; k++) v = __dsub_rn(v, __dmul_rn(A[k * LP + i], Gi[k * LP + lane]));
      Gi[i * LP + lane] = __ddiv_rn(v, A[i * LP + i]);
    }
    if (fail && lane == 0) *bad = 1;
  }
  __syncthreads();
  float* c = cm + (long long)blockIdx.x * kGramLen;
  for (int e = tid; e < T * K; e += 256) {
    double v = 0;
    for (int k = 0; k < K; k++) v = __dadd_rn(v, __dmul_rn(Bs[e / K * K + k], Gi[k * LP + e % K]));
    C1[e] = v;
    c[e] = (float)v;
    red[e] = __dmul_rn(v, Bs[e]);
  }
  __syncthreads();
  for (int e = tid; e < K * K; e += 256) {
    double v = 0;
    for (int i = 0; i < T; i++) v = __dadd_rn(v, __dmul_rn(C1[i * K + e / K], C1[i * K + e % K]));
    c[T * K + e] = (float)v;
  }
  if (tid == 0) {
    double cap = 0;
    for (int i = 0; i < T * K; i++) cap = __dadd_rn(cap, red[i]);
    loss[blockIdx.x] = T - cap;
  }
}

// dY[p][j] = -2 (sum_i V[p][i] C1[i][j] - sum_k Y[p][k] C2[k][j])
__global__ void __launch_bounds__(256) k_ln_dy(const LnPatch* __restrict__ lp, const float* __restrict__ y,
                                               const float* __restrict__ v, const float* __restrict__ cm,
                                               float* __restrict__ dy) {
  __shared__ __align__(16) LnRows rows[8];
  const LnPatch P = lp[blockIdx.y];
  const long long N = (long long)P.H * P.W;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const float* C1 = cm + (long long)blockIdx.y * kGramLen;  // [9][32]
  const float* C2 = C1 + kLnTargets * kLnOut;                  // [32][32]
  float c1[kLnTargets], c2[kLnOut];
#pragma unroll
  for (int i = 0; i < kLnTargets; i++) c1[i] = C1[i * kLnOut + lane];
#pragma unroll
  for (int k = 0; k < kLnOut; k++) c2[k] = C2[k * kLnOut + lane];
  const long long w0 = (long long)blockIdx.x * 8 + warp, nw = (long long)gridDim.x * 8;
  LnRows& r = rows[warp];
  auto count = [&](long long p) { return p < N ? (int)min(N - p, 4LL) : 0; };
  LnShare next = ln_fetch(y, v, P.off + 4 * w0, 1, count(4 * w0), lane);
  for (long long p = 4 * w0; p < N; p += 4 * nw) {
    const int n = count(p);
    ln_store(r, next, lane);
    next = ln_fetch(y, v, P.off + p + 4 * nw, 1, count(p + 4 * nw), lane);
#pragma unroll
    for (int k4 = 0; k4 < 4; k4++) {
      if (k4 >= n) break;
      float yk[kLnOut], vi[kVPitch];
      ln_row(r, k4, yk, vi);
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < kLnTargets; i++) s = fmaf(vi[i], c1[i], s);
#pragma unroll
      for (int k = 0; k < kLnOut; k++) s = fmaf(-yk[k], c2[k], s);
      dy[(P.off + p + k4) * kLnOut + lane] = -2.f * s;
    }
  }
}

// --------------------------------------------------------------- weights
// BF16 copies of every convolution's weights: wb [cout][9][cin] and the
// flipped, transposed wt [cin][9][cout] (wt[c][8 - tap][n] = W[n][tap][c]),
// both at the parameter vector's weight offsets
struct ConvOff {
  long long wo[kLnConvs];
  int cin[kLnConvs], cout[kLnConvs];
};
__global__ void k_ln_wprep(ConvOff co, const float* __restrict__ w32, bf16* __restrict__ wb,
                           bf16* __restrict__ wt) {
  const int l = blockIdx.y;
  const int ci = co.cin[l], cn = co.cout[l];
  const long long n9 = (long long)cn * 9 * ci;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n9; i += (long long)gridDim.x * blockDim.x) {
    const float v = w32[co.wo[l] + i];
    const int c = (int)(i % ci), tap = (int)((i / ci) % 9), n = (int)(i / (9 * (long long)ci));
    wb[co.wo[l] + i] = __float2bfloat16_rn(v);
    wt[co.wo[l] + ((long long)c * 9 + (8 - tap)) * cn + n] = __float2bfloat16_rn(v);
  }
}

__global__ void k_ln_adam(long long n, float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                          float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi, vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// start block: X[vec + p][j] = y[p][j] + 1e-2 * (mean |y[p][.]| + 1e-6) * u(p, j)
__device__ __forceinline__ float ln_hash(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352dU;
  x ^= x >> 15;
  x *= 0x846ca68bU;
  x ^= x >> 16;
  return (float)(x & 0xffffff) * (1.0f / 16777216.0f) - 0.5f;
}
__global__ void k_ln_start(const LnPatch* __restrict__ lp, const PatchDev* __restrict__ pd,
                           const float* __restrict__ y, float* __restrict__ X) {
  const LnPatch P = lp[blockIdx.y];
  const PatchDev D = pd[blockIdx.y];
  const int lane = threadIdx.x & 31;
  const long long w0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long p = w0; p < (long long)P.H * P.W; p += nw) {
    const float v = y[(P.off + p) * kLnOut + lane];
    float a = fabsf(v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    const float amp = 1e-2f * (a * (1.f / 32.f) + 1e-6f);
    X[(D.vec + p) * kBlk + lane] = v + amp * ln_hash((uint32_t)(p * 32 + lane) * 2654435761u + 977u);
  }
}

template <int CIN, int CO, int MODE, int C1>
cudaError_t conv_go(const LnPatch* lp, const LnTile* tiles, int ntiles, int cout, const LnIn& in, const float* dA,
                    const bf16* mask, const bf16* w, const float* bias, void* out, cudaStream_t s) {
  constexpr size_t smem = ((size_t)NHALO * (CIN + 8) + (size_t)CO * (9 * CIN + 8)) * sizeof(bf16);
  static PerDevice ready;
  const cudaError_t e = ready.once([] { return grant_smem(k_ln_conv<CIN, CO, MODE, C1>, smem); });
  if (e != cudaSuccess || ntiles == 0) return e;
  // Up to 16 input channels a tile per CTA: the weights are under 10 KB, and
  // 12-16 CTAs per SM overlap one another's staging (62 us for the three of
  // a forward of 617 kpx against 67 us persistent).  Wider layers: as many
  // CTAs as fit the SMs together, in equal shares of the tiles, so the
  // weights (up to 74 KB) are staged once (128 channels: 47 us against 69).
  const int chunks = cout / CO;
  const int fit = std::max(1, 152 * (int)std::min<size_t>(12, 227 * 1024 / (smem + 1024)) / chunks);
  const int per = CIN <= 16 ? 1 : (ntiles + fit - 1) / fit;
  k_ln_conv<CIN, CO, MODE, C1><<<dim3((ntiles + per - 1) / per, chunks), kConvThreads, smem, s>>>(
      lp, tiles, ntiles, in, dA, mask, w, bias, out, cout);
  return cudaGetLastError();
}

// the instantiations the network uses: forward (mode 0 / 1) and data
// gradient (mode 2, cin = the layer's cout, cout = its cin)
cudaError_t conv_launch(int cin, int cout, int mode, const LnPatch* lp, const LnTile* tiles, int ntiles,
                        const LnIn& in, const float* dA, const bf16* mask, const bf16* w, const float* bias,
                        void* out, cudaStream_t s) {
  const bool c16 = (cout % 32) != 0;
#define GO(CI, CO, M, C1) return conv_go<CI, CO, M, C1>(lp, tiles, ntiles, cout, in, dA, mask, w, bias, out, s)
  if (mode == 0) {
    if (c16) {
      if (cin == 16) GO(16, 16, 0, 0);
      if (cin == 48) GO(48, 16, 0, 32);
    } else {
      if (cin == 16) GO(16, 32, 0, 0);
      if (cin == 32) GO(32, 32, 0, 0);
      if (cin == 64) GO(64, 32, 0, 0);
      if (cin == 96) GO(96, 32, 0, 64);
      if (cin == 128) GO(128, 32, 0, 64);
    }
  } else if (mode == 1) {
    if (cin == 16 && !c16) GO(16, 32, 1, 0);
  } else {
    if (c16) {
      if (cin == 16) GO(16, 16, 2, 0);
      if (cin == 32) GO(32, 16, 2, 0);
    } else {
      if (cin == 32) GO(32, 32, 2, 0);
      if (cin == 64) GO(64, 32, 2, 0);
    }
  }
#undef GO
  return cudaErrorInvalidValue;
}

template <int CIN, int CC, int COUT, int WC, int C1>
cudaError_t wgrad_go(const LnPatch* lp, const LnTile* tiles, int ntiles, const float* dA, const bf16* mask,
                     const LnIn& X, float* dW, float* db, cudaStream_t s) {
  using G = WgradCfg<CIN, CC, COUT, WC>;
  static PerDevice ready;
  const cudaError_t e = ready.once([] { return grant_smem(k_ln_wgrad<CIN, CC, COUT, WC, C1>, G::smem); });
  if (e != cudaSuccess) return e;
  // about two CTAs per SM over the channel chunks; one where a thread's sums
  // take most of its registers
  constexpr int chunks = CIN / CC, per_sm = G::CPW * G::NT >= 4 ? 1 : 2;
  const dim3 grid(std::max(1, std::min(ntiles, 152 * per_sm / chunks)), chunks);
  k_ln_wgrad<CIN, CC, COUT, WC, C1><<<grid, 256, G::smem, s>>>(lp, tiles, ntiles, dA, mask, X, dW, db);
  return cudaGetLastError();
}
cudaError_t wgrad_launch(int cin, int cout, const LnPatch* lp, const LnTile* tiles, int ntiles, const float* dA,
                         const bf16* mask, const LnIn& X, float* dW, float* db, cudaStream_t s) {
  if (ntiles == 0) return cudaSuccess;
#define GO(CI, CC, CO, WC, C1) return wgrad_go<CI, CC, CO, WC, C1>(lp, tiles, ntiles, dA, mask, X, dW, db, s)
  if (cin == 16 && cout == 16) GO(16, 16, 16, 2, 0);
  if (cin == 16 && cout == 32) GO(16, 16, 32, 2, 0);
  if (cin == 32 && cout == 32) GO(32, 32, 32, 4, 0);
  if (cin == 32 && cout == 64) GO(32, 32, 64, 4, 0);
  if (cin == 64 && cout == 64) GO(64, 64, 64, 8, 0);
  if (cin == 128 && cout == 64) GO(128, 64, 64, 8, 64);
  if (cin == 96 && cout == 32) GO(96, 32, 32, 4, 64);
  if (cin == 48 && cout == 16) GO(48, 48, 16, 2, 32);
#undef GO
  return cudaErrorInvalidValue;
}

dim3 pix_grid(long long maxpix, int npatch) {
  return dim3((unsigned)std::max(1LL, std::min((maxpix + 255) / 256, 4096LL)), npatch);
}

}  // namespace

// ----------------------------------------------------------------- host
struct LearnedNet::Impl {
  size_t wo[kLnConvs], bo[kLnConvs], np = 0;
  float* w32 = nullptr;  // master weights
  float* grad = nullptr;
  float *am = nullptr, *av = nullptr;  // Adam moments
  bf16 *wb = nullptr, *wt = nullptr;   // BF16 weights, flipped-transposed BF16 weights
  bool have = false;
  std::vector<int> h, w;  // the sizes that the layout below was built for
  std::vector<LnPatch> lp[kLnLevels];
  std::vector<LnTile> lt[kLnLevels];
  long long npix[kLnLevels] = {0, 0, 0, 0}, maxpix[kLnLevels] = {0, 0, 0, 0};
  LnPatch* d_lp[kLnLevels] = {};
  LnTile* d_lt[kLnLevels] = {};
  size_t cap_lp[kLnLevels] = {}, cap_lt[kLnLevels] = {};
  // activations (BF16) and gradients (FP32), one arena each, carved per level
  bf16* act = nullptr;
  size_t cap_act = 0;
  float* gr = nullptr;
  size_t cap_gr = 0;
  float* y = nullptr;
  size_t cap_y = 0;
  double* gram = nullptr;
  float* cm = nullptr;
  double* ploss = nullptr;  // loss per patch
  int* bad = nullptr;
  size_t cap_gram = 0, cap_cm = 0, cap_ploss = 0, cap_bad = 0;
  std::vector<double> h_loss;
  // named tensors
  bf16 *X0, *A0a, *S0, *A0c, *A0d, *P0, *A1a, *S1, *A1c, *A1d, *P1, *A2a, *S2, *A2c, *A2d, *P2,
      *A3a, *A3b;
  float *dY, *dA0d, *dA0c, *dC0, *dS0, *dA0a, *dA1d, *dA1c, *dC1, *dS1, *dA1a, *dP0, *dA2d, *dA2c, *dC2, *dS2,
      *dA2a, *dP1, *dA3b, *dA3a, *dP2;
  int launches = 0;

  Impl() { conv_offsets(wo, bo, &np); }
  ~Impl() {
    void* ps[] = {w32, grad, am, av, wb, wt, act, gr, y, gram, cm, ploss, bad};
    for (void* p : ps)
      if (p) cudaFree(p);
    for (int l = 0; l < kLnLevels; l++) {
      if (d_lp[l]) cudaFree(d_lp[l]);
      if (d_lt[l]) cudaFree(d_lt[l]);
    }
  }
  cudaError_t wprep(cudaStream_t s) {
    ConvOff co;
    for (int l = 0; l < kLnConvs; l++) {
      co.wo[l] = (long long)wo[l];
      co.cin[l] = kLnNet[l].cin;
      co.cout[l] = kLnNet[l].cout;
    }
    k_ln_wprep<<<dim3(64, kLnConvs), 256, 0, s>>>(co, w32, wb, wt);
    launches++;
    return cudaGetLastError();
  }
  LnIn one(const bf16* x) const { return {x, nullptr, nullptr}; }
  // [up-sampled coarse, skip] at a level
  LnIn cat(int level, const bf16* coarse, const bf16* skip) const { return {skip, coarse, d_lp[level + 1]}; }
  cudaError_t conv(int l, int level, const LnIn& in, void* out, cudaStream_t s) {
    launches++;
    return conv_launch(kLnNet[l].cin, kLnNet[l].cout, kLnNet[l].relu ? 0 : 1, d_lp[level], d_lt[level],
                       (int)lt[level].size(), in, nullptr, nullptr, wb + wo[l], w32 + bo[l], out, s);
  }
  // backward of convolution l: dA (FP32 gradient of its output), mask (its
  // BF16 output; null for the head), X (its input); the data gradient into
  // dX unless null
  cudaError_t conv_bwd(int l, int level, const float* dA, const bf16* mask, const LnIn& X, float* dX,
                       cudaStream_t s) {
    cudaError_t e = wgrad_launch(kLnNet[l].cin, kLnNet[l].cout, d_lp[level], d_lt[level], (int)lt[level].size(), dA,
                                 mask, X, grad + wo[l], grad + bo[l], s);
    launches++;
    if (e != cudaSuccess || !dX) return e;
    launches++;
    return conv_launch(kLnNet[l].cout, kLnNet[l].cin, 2, d_lp[level], d_lt[level], (int)lt[level].size(), LnIn{},
                       dA, mask, wt + wo[l], nullptr, dX, s);
  }
};

LearnedNet::LearnedNet() : im_(new Impl()) {}
LearnedNet::~LearnedNet() = default;
bool LearnedNet::has_params() const { return im_->have; }
const std::vector<LnPatch>& LearnedNet::patches0() const { return im_->lp[0]; }
const LnPatch* LearnedNet::patches0_dev() const { return im_->d_lp[0]; }
long long LearnedNet::npix0() const { return im_->npix[0]; }
float* LearnedNet::y() { return im_->y; }
float* LearnedNet::grad() { return im_->grad; }
int LearnedNet::launches() const { return im_->launches; }

template <class T>
static cudaError_t grow_buf(T*& p, size_t& cap, size_t need) {
  if (need <= cap && p) return cudaSuccess;
  if (p) cudaFree(p);
  p = nullptr;
  cap = 0;
  cudaError_t e = cudaMalloc(&p, std::max<size_t>(need, 1) * sizeof(T));
  if (e == cudaSuccess) cap = need;
  return e;
}

cudaError_t LearnedNet::set_params(const float* hp, cudaStream_t s) {
  Impl& m = *im_;
  cudaError_t e;
  if (!m.w32) {
    size_t c = 0;
    if ((e = grow_buf(m.w32, c, m.np)) != cudaSuccess) return e;
    c = 0;
    if ((e = grow_buf(m.grad, c, m.np)) != cudaSuccess) return e;
    c = 0;
    if ((e = grow_buf(m.am, c, m.np)) != cudaSuccess) return e;
    c = 0;
    if ((e = grow_buf(m.av, c, m.np)) != cudaSuccess) return e;
    c = 0;
    if ((e = grow_buf(m.wb, c, m.np)) != cudaSuccess) return e;
    c = 0;
    if ((e = grow_buf(m.wt, c, m.np)) != cudaSuccess) return e;
  }
  if ((e = cudaMemcpyAsync(m.w32, hp, m.np * sizeof(float), cudaMemcpyHostToDevice, s)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(m.am, 0, m.np * sizeof(float), s)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(m.av, 0, m.np * sizeof(float), s)) != cudaSuccess) return e;
  if ((e = m.wprep(s)) != cudaSuccess) return e;
  m.have = true;
  return cudaSuccess;
}

cudaError_t LearnedNet::get_params(float* hp, cudaStream_t s) {
  if (!im_->have) return cudaErrorInvalidValue;
  cudaError_t e = cudaMemcpyAsync(hp, im_->w32, im_->np * sizeof(float), cudaMemcpyDeviceToHost, s);
  if (e != cudaSuccess) return e;
  return cudaStreamSynchronize(s);
}

cudaError_t LearnedNet::layout(const std::vector<int>& H, const std::vector<int>& W, cudaStream_t s) {
  Impl& m = *im_;
  const int n = (int)H.size();
  if (H == m.h && W == m.w) return cudaSuccess;  // the tables and tensors of these sizes are in place
  m.h.clear();  // until all of it is
  for (int l = 0; l < kLnLevels; l++) {
    m.lp[l].clear();
    m.lt[l].clear();
    long long off = 0, mx = 0;
    for (int i = 0; i < n; i++) {
      int h = H[i], w = W[i];
      for (int k = 0; k < l; k++) {
        h = (h + 1) / 2;
        w = (w + 1) / 2;
      }
      m.lp[l].push_back({h, w, off});
      for (int y = 0; y < h; y += TH)
        for (int x = 0; x < w; x += TW) m.lt[l].push_back({i, y, x, 0});
      off += (long long)h * w;
      mx = std::max(mx, (long long)h * w);
    }
    m.npix[l] = off;
    m.maxpix[l] = mx;
    cudaError_t e;
    if ((e = grow_buf(m.d_lp[l], m.cap_lp[l], m.lp[l].size())) != cudaSuccess) return e;
    if ((e = grow_buf(m.d_lt[l], m.cap_lt[l], std::max<size_t>(1, m.lt[l].size()))) != cudaSuccess) return e;
    if ((e = cudaMemcpyAsync(m.d_lp[l], m.lp[l].data(), m.lp[l].size() * sizeof(LnPatch), cudaMemcpyHostToDevice,
                             s)) != cudaSuccess)
      return e;
    if (!m.lt[l].empty() && (e = cudaMemcpyAsync(m.d_lt[l], m.lt[l].data(), m.lt[l].size() * sizeof(LnTile),
                                                 cudaMemcpyHostToDevice, s)) != cudaSuccess)
      return e;
  }
  // channel counts of the BF16 activations per level, then of the FP32
  // gradients; each tensor is its level's pixel count times its channels
  const long long N0 = m.npix[0], N1 = m.npix[1], N2 = m.npix[2], N3 = m.npix[3];
  const size_t act_need = N0 * (16 + 16 + 16 + 16 + 16) + N1 * (16 + 32 + 32 + 32 + 32) +
                          N2 * (32 + 64 + 64 + 64 + 64) + N3 * (64 + 64 + 64);
  const size_t gr_need = N0 * (32 + 16 + 16 + 48 + 16 + 16) + N1 * (32 + 32 + 96 + 32 + 32 + 16) +
                         N2 * (64 + 64 + 128 + 64 + 64 + 32) + N3 * (64 + 64 + 64);
  cudaError_t e;
  if ((e = grow_buf(m.act, m.cap_act, act_need)) != cudaSuccess) return e;
  if ((e = grow_buf(m.gr, m.cap_gr, gr_need)) != cudaSuccess) return e;
  if ((e = grow_buf(m.y, m.cap_y, (size_t)N0 * kLnOut)) != cudaSuccess) return e;
  if ((e = grow_buf(m.gram, m.cap_gram, (size_t)n * kGramLen)) != cudaSuccess) return e;
  if ((e = grow_buf(m.cm, m.cap_cm, (size_t)n * kGramLen)) != cudaSuccess) return e;
  if ((e = grow_buf(m.ploss, m.cap_ploss, (size_t)n)) != cudaSuccess) return e;
  if ((e = grow_buf(m.bad, m.cap_bad, 1)) != cudaSuccess) return e;
  bf16* a = m.act;
  auto A = [&](long long N, int C) {
    bf16* r = a;
    a += N * C;
    return r;
  };
  m.X0 = A(N0, 16), m.A0a = A(N0, 16), m.S0 = A(N0, 16), m.A0c = A(N0, 16), m.A0d = A(N0, 16);
  m.P0 = A(N1, 16), m.A1a = A(N1, 32), m.S1 = A(N1, 32), m.A1c = A(N1, 32), m.A1d = A(N1, 32);
  m.P1 = A(N2, 32), m.A2a = A(N2, 64), m.S2 = A(N2, 64), m.A2c = A(N2, 64), m.A2d = A(N2, 64);
  m.P2 = A(N3, 64), m.A3a = A(N3, 64), m.A3b = A(N3, 64);
  float* g = m.gr;
  auto G = [&](long long N, int C) {
    float* r = g;
    g += N * C;
    return r;
  };
  m.dY = G(N0, 32), m.dA0d = G(N0, 16), m.dA0c = G(N0, 16), m.dC0 = G(N0, 48), m.dS0 = G(N0, 16), m.dA0a = G(N0, 16);
  m.dA1d = G(N1, 32), m.dA1c = G(N1, 32), m.dC1 = G(N1, 96), m.dS1 = G(N1, 32), m.dA1a = G(N1, 32), m.dP0 = G(N1, 16);
  m.dA2d = G(N2, 64), m.dA2c = G(N2, 64), m.dC2 = G(N2, 128), m.dS2 = G(N2, 64), m.dA2a = G(N2, 64), m.dP1 = G(N2, 32);
  m.dA3b = G(N3, 64), m.dA3a = G(N3, 64), m.dP2 = G(N3, 64);
  m.h = H;
  m.w = W;
  return cudaSuccess;
}

cudaError_t LearnedNet::features(const float* d_mpb, const float* d_deg, cudaStream_t s) {
  Impl& m = *im_;
  k_ln_features<<<pix_grid(m.maxpix[0], (int)m.lp[0].size()), 256, 0, s>>>(m.d_lp[0], d_mpb, d_deg, m.X0);
  m.launches++;
  return cudaGetLastError();
}

cudaError_t LearnedNet::features_from(const PatchDev* patches, const float* d_mpb, const float* d_deg,
                                      cudaStream_t s) {
  Impl& m = *im_;
  k_ln_features_from<<<pix_grid(m.maxpix[0], (int)m.lp[0].size()), 256, 0, s>>>(m.d_lp[0], patches, d_mpb, d_deg,
                                                                                m.X0);
  m.launches++;
  return cudaGetLastError();
}

cudaError_t LearnedNet::forward(cudaStream_t s, float* out) {
  Impl& m = *im_;
  if (!m.have) return cudaErrorInvalidValue;
  const int np = (int)m.lp[0].size();
  cudaError_t e;
#define CKE(x)                              \
  do {                                      \
    if ((e = (x)) != cudaSuccess) return e; \
  } while (0)
  auto pool = [&](int l, int C, const bf16* in, bf16* out) {
    k_ln_pool<<<pix_grid(m.maxpix[l + 1] * (C / 8), np), 256, 0, s>>>(m.d_lp[l], m.d_lp[l + 1], np, C, in, out);
    m.launches++;
    return cudaGetLastError();
  };
  CKE(m.conv(0, 0, m.one(m.X0), m.A0a, s));
  CKE(m.conv(1, 0, m.one(m.A0a), m.S0, s));
  CKE(pool(0, 16, m.S0, m.P0));
  CKE(m.conv(2, 1, m.one(m.P0), m.A1a, s));
  CKE(m.conv(3, 1, m.one(m.A1a), m.S1, s));
  CKE(pool(1, 32, m.S1, m.P1));
  CKE(m.conv(4, 2, m.one(m.P1), m.A2a, s));
  CKE(m.conv(5, 2, m.one(m.A2a), m.S2, s));
  CKE(pool(2, 64, m.S2, m.P2));
  CKE(m.conv(6, 3, m.one(m.P2), m.A3a, s));
  CKE(m.conv(7, 3, m.one(m.A3a), m.A3b, s));
  CKE(m.conv(8, 2, m.cat(2, m.A3b, m.S2), m.A2c, s));
  CKE(m.conv(9, 2, m.one(m.A2c), m.A2d, s));
  CKE(m.conv(10, 1, m.cat(1, m.A2d, m.S1), m.A1c, s));
  CKE(m.conv(11, 1, m.one(m.A1c), m.A1d, s));
  CKE(m.conv(12, 0, m.cat(0, m.A1d, m.S0), m.A0c, s));
  CKE(m.conv(13, 0, m.one(m.A0c), m.A0d, s));
  CKE(m.conv(14, 0, m.one(m.A0d), out ? out : m.y, s));
  return cudaSuccess;
}

// k_ln_solve on the host, for one patch: the same operations in the same
// order (the host's code is compiled without contraction); false where the
// regularised Gram matrix is not positive definite
static bool ln_solve_host(const double* g, float* cm, double* loss) {
  constexpr int K = kLnOut, T = kLnTargets;
  double A[K][K], Gi[K][K] = {}, C1[T * K];
  const double* B = g + K * K;
  double tr = 0;
  for (int i = 0; i < K; i++) tr += g[i * K + i];
  const double eps = 1e-4 * tr / K + 1e-30;
  for (int i = 0; i < K; i++)
    for (int j = 0; j < K; j++) A[i][j] = g[i * K + j] + (i == j ? eps : 0.0);
  for (int i = 0; i < K; i++) Gi[i][i] = 1.0;
  for (int j = 0; j < K; j++) {  // A becomes L, Gi becomes L^-1
    if (!(A[j][j] > 0)) return false;
    const double s = std::sqrt(A[j][j]);
    A[j][j] = s;
    for (int r = j + 1; r < K; r++) A[r][j] /= s;
    for (int q = 0; q <= j; q++) Gi[j][q] /= s;
    for (int r = j + 1; r < K; r++) {
      for (int q = j + 1; q <= r; q++) A[r][q] -= A[r][j] * A[q][j];
      for (int q = 0; q <= j; q++) Gi[r][q] -= A[r][j] * Gi[j][q];
    }
  }
  for (int i = K - 1; i >= 0; i--) {  // (L L^T)^-1
    for (int k = i + 1; k < K; k++)
      for (int c = 0; c < K; c++) Gi[i][c] -= A[k][i] * Gi[k][c];
    for (int c = 0; c < K; c++) Gi[i][c] /= A[i][i];
  }
  double cap = 0;
  for (int i = 0; i < T; i++)
    for (int j = 0; j < K; j++) {
      double v = 0;
      for (int k = 0; k < K; k++) v += B[i * K + k] * Gi[k][j];
      C1[i * K + j] = v;
      cm[i * K + j] = (float)v;
      cap += v * B[i * K + j];
    }
  for (int a = 0; a < K; a++)
    for (int b = 0; b < K; b++) {
      double v = 0;
      for (int i = 0; i < T; i++) v += C1[i * K + a] * C1[i * K + b];
      cm[T * K + a * K + b] = (float)v;
    }
  *loss = T - cap;
  return true;
}

// Gradients of up to this many patches solve on the host: a round trip and
// about 17 us a patch against the 147 us of k_ln_solve's chain.  Microseconds
// of one gradient of 64^2 patches, host / device: 1 patch 648 / 771 (48^2),
// 4 patches 711 / 806, 8 patches 812 / 851, 10 patches 852 / 870, 12 patches
// 905 / 890, 16 patches 1015 / 940.
constexpr int kHostSolve = 8;

cudaError_t LearnedNet::loss_backward(const float* d_v, double* loss, cudaStream_t s) {
  Impl& m = *im_;
  if (!m.have) return cudaErrorInvalidValue;
  const int np = (int)m.lp[0].size();
  cudaError_t e;
  // the subspace loss and its gradient with respect to y
  CKE(cudaMemsetAsync(m.gram, 0, (size_t)np * kGramLen * sizeof(double), s));
  k_ln_gram<<<dim3((unsigned)std::max(1LL, std::min(m.maxpix[0] / 2048 + 1, 512LL)), np), 256, 0, s>>>(
      m.d_lp[0], m.y, d_v, m.gram);
  m.launches++;
  CKE(cudaGetLastError());
  const bool on_host = np <= kHostSolve;
  m.h_loss.resize(np);
  if (on_host) {
    std::vector<double> g((size_t)np * kGramLen);
    std::vector<float> c((size_t)np * kGramLen);
    CKE(cudaMemcpyAsync(g.data(), m.gram, np * kGramLen * sizeof(double), cudaMemcpyDeviceToHost, s));
    CKE(cudaStreamSynchronize(s));
    for (int p = 0; p < np; p++)
      if (!ln_solve_host(&g[(size_t)p * kGramLen], &c[(size_t)p * kGramLen], &m.h_loss[p]))
        return cudaErrorInvalidValue;
    CKE(cudaMemcpyAsync(m.cm, c.data(), np * kGramLen * sizeof(float), cudaMemcpyHostToDevice, s));
  } else {
    CKE(cudaMemsetAsync(m.bad, 0, sizeof(int), s));
    k_ln_solve<<<np, 256, 0, s>>>(m.gram, m.cm, m.ploss, m.bad);
    m.launches++;
    CKE(cudaGetLastError());
  }
  k_ln_dy<<<dim3((unsigned)std::max(1LL, std::min(m.maxpix[0] / 512 + 1, 1024LL)), np), 256, 0, s>>>(
      m.d_lp[0], m.y, d_v, m.cm, m.dY);
  m.launches++;
  CKE(cudaGetLastError());
  // backward through the network
  CKE(cudaMemsetAsync(m.grad, 0, m.np * sizeof(float), s));
  auto pool_bwd = [&](int l, int C, const float* dP, float* dS) {
    k_ln_pool_bwd<<<pix_grid(m.maxpix[l] * C / 8, np), 256, 0, s>>>(m.d_lp[l], m.d_lp[l + 1], C, dP, dS);
    m.launches++;
    return cudaGetLastError();
  };
  auto upcat_bwd = [&](int l, int C1c, int C2c, const float* dC, float* dcoarse, float* dskip) {
    k_ln_upcat_bwd_coarse<<<pix_grid(m.maxpix[l + 1] * C1c / 8, np), 256, 0, s>>>(m.d_lp[l], m.d_lp[l + 1], C1c,
                                                                                   C2c, dC, dcoarse);
    k_ln_upcat_bwd_skip<<<pix_grid(m.maxpix[l] * C2c / 8, np), 256, 0, s>>>(m.d_lp[l], C1c, C2c, dC, dskip);
    m.launches += 2;
    return cudaGetLastError();
  };
  CKE(m.conv_bwd(14, 0, m.dY, nullptr, m.one(m.A0d), m.dA0d, s));
  CKE(m.conv_bwd(13, 0, m.dA0d, m.A0d, m.one(m.A0c), m.dA0c, s));
  CKE(m.conv_bwd(12, 0, m.dA0c, m.A0c, m.cat(0, m.A1d, m.S0), m.dC0, s));
  CKE(upcat_bwd(0, 32, 16, m.dC0, m.dA1d, m.dS0));
  CKE(m.conv_bwd(11, 1, m.dA1d, m.A1d, m.one(m.A1c), m.dA1c, s));
  CKE(m.conv_bwd(10, 1, m.dA1c, m.A1c, m.cat(1, m.A2d, m.S1), m.dC1, s));
  CKE(upcat_bwd(1, 64, 32, m.dC1, m.dA2d, m.dS1));
  CKE(m.conv_bwd(9, 2, m.dA2d, m.A2d, m.one(m.A2c), m.dA2c, s));
  CKE(m.conv_bwd(8, 2, m.dA2c, m.A2c, m.cat(2, m.A3b, m.S2), m.dC2, s));
  CKE(upcat_bwd(2, 64, 64, m.dC2, m.dA3b, m.dS2));
  CKE(m.conv_bwd(7, 3, m.dA3b, m.A3b, m.one(m.A3a), m.dA3a, s));
  CKE(m.conv_bwd(6, 3, m.dA3a, m.A3a, m.one(m.P2), m.dP2, s));
  CKE(pool_bwd(2, 64, m.dP2, m.dS2));
  CKE(m.conv_bwd(5, 2, m.dS2, m.S2, m.one(m.A2a), m.dA2a, s));
  CKE(m.conv_bwd(4, 2, m.dA2a, m.A2a, m.one(m.P1), m.dP1, s));
  CKE(pool_bwd(1, 32, m.dP1, m.dS1));
  CKE(m.conv_bwd(3, 1, m.dS1, m.S1, m.one(m.A1a), m.dA1a, s));
  CKE(m.conv_bwd(2, 1, m.dA1a, m.A1a, m.one(m.P0), m.dP0, s));
  CKE(pool_bwd(0, 16, m.dP0, m.dS0));
  CKE(m.conv_bwd(1, 0, m.dS0, m.S0, m.one(m.A0a), m.dA0a, s));
  CKE(m.conv_bwd(0, 0, m.dA0a, m.A0a, m.one(m.X0), nullptr, s));
  if (!on_host) {
    int bad = 0;
    CKE(cudaMemcpyAsync(m.h_loss.data(), m.ploss, np * sizeof(double), cudaMemcpyDeviceToHost, s));
    CKE(cudaMemcpyAsync(&bad, m.bad, sizeof(int), cudaMemcpyDeviceToHost, s));
    CKE(cudaStreamSynchronize(s));
    if (bad) return cudaErrorInvalidValue;  // a patch's Gram matrix is not positive definite
  }
  *loss = 0;
  for (double l : m.h_loss) *loss += l;
#undef CKE
  return cudaSuccess;
}

cudaError_t LearnedNet::adam(float lr, float b1, float b2, float eps, int t, cudaStream_t s) {
  Impl& m = *im_;
  if (!m.have) return cudaErrorInvalidValue;
  const float c1 = 1.f - powf(b1, (float)t), c2 = 1.f - powf(b2, (float)t);
  k_ln_adam<<<256, 256, 0, s>>>((long long)m.np, m.w32, m.grad, m.am, m.av, lr, b1, b2, eps, c1, c2);
  m.launches++;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return m.wprep(s);
}

cudaError_t ln_launch_start(const LnPatch* lp, const PatchDev* patches, int npatch, int maxN, const float* y,
                            float* X, cudaStream_t s) {
  k_ln_start<<<pix_grid((long long)maxN * 32 / 8, npatch), 256, 0, s>>>(lp, patches, y, X);
  return cudaGetLastError();
}

}  // namespace gpb
