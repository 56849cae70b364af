// k_block.cu -- block kernels of the Chebyshev-filtered subspace iteration
// (the warm-started eigensolver) for A = I - D^-1/2 W D^-1/2 (sm_103a).
//
// A block of kBlk = 32 vectors is stored pixel-major ([vec][32] floats) in the
// padded vector layout, so every stencil neighbour of a pixel is one
// contiguous 128-byte row; the operator of the block kernels holds one full
// stencil row per pixel, tile by tile in the order the step loads it
// (cf_full).
//
//   cf_step    Y' = alpha (A Y) + beta Y + gamma X   (scaled Chebyshev
//              recurrence, Zhou & Saad 2007; with alpha=1, beta=gamma=0 it
//              is the plain block SpMV)
//   cf_gram    G = U^T V per patch (32 x 32), FP32 FMA runs folded into
//              float-float sums, summed across CTAs by cf_gram_sum
//   cf_rotate  U <- U M (32 x 32 per patch), optionally V <- V M too
//   cf_resid   |A x_c - theta_c x_c|^2 per column
//   cf_extract the first nvec columns into separate vectors (sPb layout)
//
// Reference: the eigensolver of damascene/src/noReorthog/lanczos.cu and
// src/spectralPb.cpp:221-245 define the problem; the block method is this
// project's own.
#include <stdint.h>
#include <stdio.h>

#include <algorithm>
#include <stdlib.h>

#include "f32x2.h"
#include "gpb_internal.h"
#include "k_block.h"
#include "k_eig.h"
#include "overlap.h"
#include "per_device.h"

namespace gpb {

// radius-5 disk offsets in scanline order (dy, then dx, ascending): the
// upper half -- after the centre -- numbered k = 0..39 as the a_up planes
__host__ __device__ constexpr bool in_disk(int dy, int dx) {
  return dy * dy + dx * dx <= kStencilR * kStencilR;
}
__host__ __device__ constexpr int disk_half_width(int dy) {  // floor(sqrt(25 - dy^2))
  return dy < 0 ? disk_half_width(-dy) : dy == 0 ? 5 : dy <= 3 ? 4 : dy == 4 ? 3 : 0;
}
__host__ __device__ constexpr int upper_rows_before(int dy) {  // offsets in rows 1..dy-1
  return dy <= 1 ? 0 : upper_rows_before(dy - 1) + 2 * disk_half_width(dy - 1) + 1;
}
__host__ __device__ constexpr int upper_k(int dy, int dx) {
  return dy == 0 ? dx - 1 : kStencilR + upper_rows_before(dy) + dx + disk_half_width(dy);
}
static_assert(upper_k(0, 1) == 0 && upper_k(1, -4) == 5 && upper_k(5, 0) == kUpper - 1, "upper offset numbering");


__constant__ int c_bup_dy[kUpper], c_bup_dx[kUpper];

void upload_block(const HostTables& t, cudaStream_t s) {
  int dy[kUpper], dx[kUpper];
  for (int j = 0; j < kUpper; j++) {
    dy[j] = t.sdy[kStencilN / 2 + 1 + j];
    dx[j] = t.sdx[kStencilN / 2 + 1 + j];
    if (upper_k(dy[j], dx[j]) != j) {  // cf_step numbers the offsets at compile time
      fprintf(stderr, "gpb: stencil offset table out of scanline order at %d\n", j);
      abort();
    }
  }
  cudaMemcpyToSymbolAsync(c_bup_dy, dy, sizeof(dy), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_bup_dx, dx, sizeof(dx), 0, cudaMemcpyHostToDevice, s);
}

// ------------------------------------------------------------ Chebyshev step
// The operator of a level is stored per 16 x 16 pixel tile (the tiles of the
// 16 x 16 work list, in its order), ready for the step's loads: 4 consecutive
// stencil coefficients of a pixel are one 16-byte slot, and a tile is [chunk
// of 4 offsets][slot of 256].  A warp of the step owns 2 tile rows, a
// quarter-warp 2 x 4 pixels of them, a lane 4 block columns of these 8
// pixels.  Slot (w, k, q) = 32 w + 4 k + q holds pixel k (row k / 4, column
// k % 4) of quarter q of warp w, so the four quarters' coefficients of a load
// are 64 contiguous bytes, and a chunk of a tile is one contiguous copy.
constexpr int kTilePx = kStepTile * kStepTile;

// the radius-5 disk of the fine level (81 offsets in scanline order, rows
// padded to 84 floats = 21 x 16 bytes) and the 7 x 7 square of the coarse one
template <int NCOEF_, int R_>
struct StencilBase {
  static constexpr int R = R_, NC = NCOEF_;
};
struct DiskStencil : StencilBase<84, kStencilR> {
  static constexpr int N = kStencilN;
  __host__ __device__ static constexpr bool in(int dy, int dx) { return in_disk(dy, dx); }
  __host__ __device__ static constexpr int rows_before(int dy) {  // offsets in rows -R..dy-1
    return dy <= -R ? 0 : rows_before(dy - 1) + 2 * disk_half_width(dy - 1) + 1;
  }
  __host__ __device__ static constexpr int index(int dy, int dx) { return rows_before(dy) + dx + disk_half_width(dy); }
};
struct SquareStencil : StencilBase<52, kCR> {
  static constexpr int N = kCN;
  __host__ __device__ static constexpr bool in(int dy, int dx) {
    return dy >= -R && dy <= R && dx >= -R && dx <= R;
  }
  __host__ __device__ static constexpr int index(int dy, int dx) { return (dy + R) * (2 * R + 1) + dx + R; }
};
static_assert(DiskStencil::index(0, 0) == kStencilN / 2 && DiskStencil::index(kStencilR, 0) == kStencilN - 1,
              "disk numbering");
static_assert(SquareStencil::index(kCR, kCR) == kCN - 1, "square numbering");
static_assert(DiskStencil::NC == kFullNC && SquareStencil::NC == kCoarseNC, "row widths");

// Shared memory of the step for WARPS consumer warps of SBR tile rows each:
// two stages of Y rows with their halo, and a ring of coefficient groups.
template <class S, int WARPS, int SBR>
struct StepSmem {
  static constexpr int ROWS = WARPS * SBR;
  static constexpr int PH = ROWS + 2 * S::R, PW = kStepTile + 2 * S::R;
  static constexpr int NCH = S::NC / 4, GC = 3, NG = (NCH + GC - 1) / GC;  // chunks, chunks per group, groups
  static constexpr int RING = 4;
  static constexpr size_t y_bytes = (size_t)PH * PW * kBlk * sizeof(float);
  static constexpr size_t chunk = (size_t)ROWS * kStepTile * 16;
  static constexpr size_t group = GC * chunk;
  static constexpr size_t bars = 2 * y_bytes + RING * group;  // tile records, mbarriers
  static constexpr size_t bytes = bars + 256;
  static_assert(y_bytes % 128 == 0 && group % 128 == 0, "alignment");
  static_assert(bytes <= 232448, "shared memory per CTA");
};

// what the Y producer tells the consumers about the tile in a stage
struct StepMeta {
  int end;        // 1: no more tiles for this CTA
  int W, H, y0;
  long long vec;
  int x0, pad;
  float cx, cy, cz, pad2;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// global -> shared bulk copy: both addresses 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
// polls of the tile's barrier before a CTA gives up (each poll may suspend
// the thread for a short hardware-defined time; the copies take microseconds)
constexpr int kBarSpin = 1 << 20;
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (int it = 0; it < kBarSpin; it++)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

template <int K>
__device__ __forceinline__ float f4get(const float4& v) {
  if constexpr (K == 0) return v.x;
  else if constexpr (K == 1) return v.y;
  else if constexpr (K == 2) return v.z;
  else return v.w;
}

// The coefficient ring as a consumer warp sees it.  Group g of a tile is
// waited for when the warp's first pixel reaches its first chunk and released
// when the last pixel has loaded its last chunk; both places are known at
// compile time.
struct StepRing {
  unsigned char* base;   // the lane's slot of pixel 0 in ring place 0
  uint64_t *full, *empty;
  unsigned n0;           // groups consumed before this tile
  bool bad;              // a wait gave up: no further waits, the results are dropped
};

constexpr int SB_C = 4;  // a quarter-warp's pixels: SBR rows of 4

// one staged position (RY, DX) relative to the quarter's block origin: the
// value of this lane's columns there, times the coefficient of every block
// pixel whose stencil covers it
// C (compensated): the terms are summed by FMA in groups of four (grp) and
// each group is folded into a float-float (acc, lo) by an exact TwoSum,
// which removes the accumulation error of the 81-term sum -- the term that
// dominates near an eigenvector, where the diagonal and the off-diagonal
// sum nearly cancel -- down to the groups' own four-term rounding, at about
// a third of the cost of a TwoSum per term; used for the Rayleigh-Ritz
// products and residuals, not the filter
template <class S, int WARPS, int SBR, bool C, int RY, int DX, int I>
__device__ __forceinline__ void step_pixels(StepRing& ring, const unsigned char* (&gb)[StepSmem<S, WARPS, SBR>::NG],
                                            const F2 (&v)[2], float4 (&cw)[SBR * SB_C], F2 (&acc)[SBR * SB_C][2],
                                            F2 (&lo)[SBR * SB_C][2], F2 (&grp)[SBR * SB_C][2]) {
  using SM = StepSmem<S, WARPS, SBR>;
  if constexpr (I < SBR * SB_C) {
    constexpr int bi = I / SB_C, bj = I % SB_C;
    if constexpr (S::in(RY - bi, DX - bj)) {
      constexpr int idx = S::index(RY - bi, DX - bj), ch = idx / 4, g = ch / SM::GC;
      // a pixel meets its offsets in scanline order, so chunk idx / 4 is
      // first needed at idx % 4 == 0; pixel 0 is the first to get there
      // (smallest row and column), pixel SBR * SB_C - 1 the last
      if constexpr (idx % 4 == 0) {
        if constexpr (I == 0 && ch % SM::GC == 0) {
          const unsigned n = ring.n0 + g;
          if (!ring.bad) ring.bad = !mbar_wait(ring.full + n % SM::RING, (n / SM::RING) & 1);
          gb[g] = ring.base + (n % SM::RING) * SM::group;
        }
        cw[I] = *(const float4*)(gb[g] + (ch % SM::GC) * SM::chunk + I * 64);
        if constexpr (I == SBR * SB_C - 1 && (ch % SM::GC == SM::GC - 1 || ch == SM::NCH - 1)) {
          __syncwarp();
          if ((threadIdx.x & 31) == 0) mbar_arrive(ring.empty + (ring.n0 + g) % SM::RING);
        }
      }
      const float c1 = f4get<idx % 4>(cw[I]);
      const F2 cf = f2(c1, c1);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        if constexpr (C) {
          grp[I][h] = f2_fma(cf, v[h], grp[I][h]);
          // a pixel's offsets run 0 .. N-1 in order: fold after every fourth
          if constexpr (idx % 4 == 3 || idx == S::N - 1) {
            const F2 t = f2_add(acc[I][h], grp[I][h]), z = f2_sub(t, acc[I][h]);
            lo[I][h] = f2_add(lo[I][h], f2_add(f2_sub(acc[I][h], f2_sub(t, z)), f2_sub(grp[I][h], z)));
            acc[I][h] = t;
            grp[I][h] = f2(0.f, 0.f);
          }
        } else {
          acc[I][h] = f2_fma(cf, v[h], acc[I][h]);
        }
      }
    }
    step_pixels<S, WARPS, SBR, C, RY, DX, I + 1>(ring, gb, v, cw, acc, lo, grp);
  }
}

// whether position P of the block's window feeds any of its pixels
template <class S, int SBR>
__host__ __device__ constexpr bool step_used(int P) {
  const int NX = SB_C + 2 * S::R, RY = P / NX - S::R, DX = P % NX - S::R;
  for (int i = 0; i < SBR; i++)
    for (int j = 0; j < SB_C; j++)
      if (S::in(RY - i, DX - j)) return true;
  return false;
}
template <class S, int SBR>
__host__ __device__ constexpr int step_next(int P) {  // the first used position from P on
  const int n = (SBR + 2 * S::R) * (SB_C + 2 * S::R);
  while (P < n && !step_used<S, SBR>(P)) P++;
  return P;
}
template <class S, int WARPS, int SBR, int P>
__device__ __forceinline__ float4 step_value(const float* __restrict__ ys) {
  constexpr int NX = SB_C + 2 * S::R;
  return *(const float4*)(ys + (P / NX * StepSmem<S, WARPS, SBR>::PW + P % NX) * kBlk);
}
// positions P, ... in scanline order; v is P's value, loaded one position ahead
template <class S, int WARPS, int SBR, bool C, int P>
__device__ __forceinline__ void step_positions(const float* __restrict__ ys, float4 v4, StepRing& ring,
                                               const unsigned char* (&gb)[StepSmem<S, WARPS, SBR>::NG],
                                               float4 (&cw)[SBR * SB_C], F2 (&acc)[SBR * SB_C][2], F2 (&lo)[SBR * SB_C][2],
                                               F2 (&grp)[SBR * SB_C][2]) {
  constexpr int NY = SBR + 2 * S::R, NX = SB_C + 2 * S::R;
  if constexpr (P < NY * NX) {
    constexpr int RY = P / NX - S::R, DX = P % NX - S::R, PN = step_next<S, SBR>(P + 1);
    float4 vn = v4;
    if constexpr (PN < NY * NX) vn = step_value<S, WARPS, SBR, PN>(ys);
    const F2 v[2] = {f2(v4.x, v4.y), f2(v4.z, v4.w)};
    step_pixels<S, WARPS, SBR, C, RY, DX, 0>(ring, gb, v, cw, acc, lo, grp);
    step_positions<S, WARPS, SBR, C, PN>(ys, vn, ring, gb, cw, acc, lo, grp);
  }
}

// Persistent, warp-specialised: one CTA per SM walks its share of the tile
// list.  Warp WARPS (one lane) streams the Y rows: for each active tile it
// waits until the consumers have released the stage, writes the tile record
// and issues bulk copies against the stage's "full" mbarrier, so tile i+1's
// rows arrive while tile i is computed.  Warp WARPS + 1 (one lane) streams
// the coefficients through a ring of groups of GC chunks.  Warps
// 0 .. WARPS-1 consume: wait "full", fetch X into registers, run the stencil
// on their 2 rows, write the outputs and arrive on the stage's "empty"
// mbarrier.  Every wait is bounded; a wait that gives up sets *a.err and ends
// the thread's work.
//
// What bounds it: HBM (720 B / px of the fine level = 118 us for 1.11 Mpx at
// the copy rate), the shared-memory pipe (111 us of wavefronts) and the FMA
// pipe, about evenly; two warps per scheduler leave some of their latency
// uncovered.  A 16-byte shared load takes 4 cycles for 32 distinct addresses
// and 2 for up to 4 (both measured), so a coefficient load that serves four
// quarters of 4 columns each feeds 16 FMAs per 2 cycles, twice as many as
// with half-warps of 2 columns; the pixel block of 2 x 4 keeps the value loads
// at 16 per pixel, and the packed FMAs halve the instructions.
// Measured, 16 patches of 266^2: 171 us per launch over all patches, 4.8 TB/s
// of DRAM traffic, from 203 us with 8 x 16 tiles, half-warps and scalar FMAs
// (187 us with scalar FMAs in this layout); same results to the bit.
// SBR = 2 (16 x 16 tiles) reads a third less halo than SBR = 1 (8 x 16) and
// loads each value for twice the pixels.  SBR = 1 is for launches whose tiles
// do not fill the SMs: half the work in each warp's chain (10 against 12.5 us a
// launch at 20 tiles, 202 against 175 us at 4624, 33 against 29 at 600).
constexpr int kStepWarps = 8;
template <class S, bool C, int WARPS, int SBR>
__global__ void __launch_bounds__((WARPS + 2) * 32, 1) cf_step_t(BlkArgs a, const int4* __restrict__ work, int nwork,
                                                                 const float* __restrict__ Y,
                                                                 const float* __restrict__ X,
                                                                 float* __restrict__ out, int step) {
  using SM = StepSmem<S, WARPS, SBR>;
  constexpr int SB_N = SBR * SB_C, SUB = kStepTile / SM::ROWS;  // SUB: this kernel's tiles per work entry
  extern __shared__ __align__(128) unsigned char smem[];
  StepMeta* meta = (StepMeta*)(smem + SM::bars);  // [2]
  uint64_t* yfull = (uint64_t*)(smem + SM::bars + 128);
  uint64_t* yempty = yfull + 2;
  uint64_t* cfull = yempty + 2;
  uint64_t* cempty = cfull + SM::RING;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; i++) {
      mbar_init(yfull + i, 1);
      mbar_init(yempty + i, WARPS);
    }
    for (int i = 0; i < SM::RING; i++) {
      mbar_init(cfull + i, 1);
      mbar_init(cempty + i, WARPS);
    }
  }
  __syncthreads();
  // the next step's CTAs may set up and fetch coefficients as this one's end
  overlap_release();
  if (warp >= WARPS) {  // ------------------------------------- producers
    if (lane != 0) return;
    if (warp == WARPS) overlap_wait();  // Y; the operator does not change within a chain of steps
    int i = 0;
    for (int t = blockIdx.x; t < nwork * SUB; t += gridDim.x) {
      const int4 w = work[t / SUB];
      const int sub = t % SUB, y0 = w.y + sub * SM::ROWS;
      if (!a.active[w.x]) continue;
      const PatchDev P = a.patches[w.x];
      if (y0 >= P.H) continue;
      if (warp == WARPS) {
        const int st = i & 1;
        if (i >= 2 && !mbar_wait(yempty + st, ((i >> 1) - 1) & 1)) {
          atomicExch(a.err, 1);
          return;
        }
        const float3 co = a.coef[(long long)w.x * a.max_steps + step];
        StepMeta& m = meta[st];
        m.end = 0;
        m.W = P.W;
        m.H = P.H;
        m.y0 = y0;
        m.x0 = w.z;
        m.vec = P.vec;
        m.cx = co.x;
        m.cy = co.y;
        m.cz = co.z;
        // rows past the patch's last row (+ the radius) feed no in-patch pixel
        const int ny = min(SM::ROWS, P.H - y0) + 2 * S::R;
        constexpr uint32_t yrow = SM::PW * kBlk * sizeof(float);
        unsigned char* ys = smem + st * SM::y_bytes;
        mbar_expect_tx(yfull + st, (uint32_t)ny * yrow);
        for (int r = 0; r < ny; r++)
          bulk_g2s(ys + (size_t)r * yrow, Y + (P.vec + (long long)(y0 - S::R + r) * P.W + (w.z - S::R)) * kBlk, yrow,
                   yfull + st);
      } else {
        const float4* src = (const float4*)a.afull + (long long)w.w * SM::NCH * kTilePx + sub * SM::ROWS * kStepTile;
        for (int g = 0; g < SM::NG; g++) {
          const int n = i * SM::NG + g, pl = n % SM::RING;
          if (n >= SM::RING && !mbar_wait(cempty + pl, (n / SM::RING - 1) & 1)) {
            atomicExch(a.err, 1);
            return;
          }
          const int nch = min(SM::GC, SM::NCH - g * SM::GC);
          unsigned char* dst = smem + 2 * SM::y_bytes + pl * SM::group;
          mbar_expect_tx(cfull + pl, (uint32_t)(nch * SM::chunk));
          if constexpr (SUB == 1) {
            bulk_g2s(dst, src + (long long)g * SM::GC * kTilePx, (uint32_t)(nch * SM::chunk), cfull + pl);
          } else {
            for (int c = 0; c < nch; c++)
              bulk_g2s(dst + c * SM::chunk, src + (long long)(g * SM::GC + c) * kTilePx, (uint32_t)SM::chunk,
                       cfull + pl);
          }
        }
      }
      i++;
    }
    if (warp == WARPS) {
      const int st = i & 1;
      if (i >= 2 && !mbar_wait(yempty + st, ((i >> 1) - 1) & 1)) {
        atomicExch(a.err, 1);
        return;
      }
      meta[st].end = 1;
      mbar_arrive(yfull + st);
    }
    return;
  }
  // ------------------------------------------------------------ consumers
  // warp: tile rows SBR warp ..; quarter: columns 4 quarter .. + 3; lane:
  // block columns col .. col + 3
  const int quarter = lane >> 3, by = SBR * warp, bx = SB_C * quarter, col = 4 * (lane & 7);
  StepRing ring;
  // the slot of the quarter's first pixel, which is pixel 0 or 4 of its row pair
  ring.base = smem + 2 * SM::y_bytes + (32 * (by >> 1) + 16 * (by & 1) + quarter) * 16;
  ring.full = cfull;
  ring.empty = cempty;
  ring.n0 = 0;
  ring.bad = false;
  overlap_wait();  // X, and the readers of out
  for (int i = 0;; i++, ring.n0 += SM::NG) {
    const int st = i & 1;
    if (!mbar_wait(yfull + st, (i >> 1) & 1)) {
      if (lane == 0) atomicExch(a.err, 1);
      return;
    }
    const StepMeta m = meta[st];
    if (m.end) return;
    if (m.y0 + by >= m.H) {  // no row of this warp is in the patch
      for (int g = 0; g < SM::NG; g++) {
        const unsigned n = ring.n0 + g;
        if (!mbar_wait(cfull + n % SM::RING, (n / SM::RING) & 1)) {
          if (lane == 0) atomicExch(a.err, 1);
          return;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(cempty + n % SM::RING);
      }
      if (lane == 0) mbar_arrive(yempty + st);
      continue;
    }
    const float* ys = (const float*)(smem + st * SM::y_bytes) + (by * SM::PW + bx) * kBlk + col;
    const long long q0 = (m.vec + (long long)(m.y0 + by) * m.W + m.x0 + bx) * kBlk + col;
    // the previous iterate's values, fetched now so the loads overlap the
    // stencil (the compensated products, whose accumulators take the
    // registers, have none)
    float4 xr[SB_N];
    auto fetch_x = [&]() {
#pragma unroll
      for (int k = 0; k < SB_N; k++) {
        const bool ok = m.cz != 0.f && m.y0 + by + k / SB_C < m.H && m.x0 + bx + k % SB_C < m.W;
        xr[k] = ok ? __ldcs((const float4*)(X + q0 + ((long long)(k / SB_C) * m.W + k % SB_C) * kBlk))
                   : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    if constexpr (!C) fetch_x();
    F2 acc[SB_N][2], lo[SB_N][2], grp[SB_N][2];
    float4 cw[SB_N];
    const unsigned char* gb[SM::NG];
#pragma unroll
    for (int k = 0; k < SB_N; k++)
#pragma unroll
      for (int h = 0; h < 2; h++) acc[k][h] = lo[k][h] = grp[k][h] = f2(0.f, 0.f);
    constexpr int P0 = step_next<S, SBR>(0);
    step_positions<S, WARPS, SBR, C, P0>(ys, step_value<S, WARPS, SBR, P0>(ys), ring, gb, cw, acc, lo, grp);
    if (ring.bad) {
      if (lane == 0) atomicExch(a.err, 1);
      return;
    }
    if constexpr (C) fetch_x();
#pragma unroll
    for (int k = 0; k < SB_N; k++) {
      if (m.y0 + by + k / SB_C >= m.H || m.x0 + bx + k % SB_C >= m.W) continue;
      const float4 y4 = *(const float4*)(ys + ((k / SB_C + S::R) * SM::PW + k % SB_C + S::R) * kBlk);
      const float yc[4] = {y4.x, y4.y, y4.z, y4.w}, xc[4] = {xr[k].x, xr[k].y, xr[k].z, xr[k].w};
      const float2 p0 = f2_split(C ? f2_add(acc[k][0], lo[k][0]) : acc[k][0]);
      const float2 p1 = f2_split(C ? f2_add(acc[k][1], lo[k][1]) : acc[k][1]);
      const float as[4] = {p0.x, p0.y, p1.x, p1.y};
      float r[4];
#pragma unroll
      for (int c = 0; c < 4; c++) {
        const float a0 = as[c];
        r[c] = fmaf(m.cy, yc[c], __fmul_rn(m.cx, a0));
        if (m.cz != 0.f) r[c] = fmaf(m.cz, xc[c], r[c]);
      }
      *(float4*)(out + q0 + ((long long)(k / SB_C) * m.W + k % SB_C) * kBlk) = make_float4(r[0], r[1], r[2], r[3]);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(yempty + st);
  }
}

// The stencil rows of the fine operator from its symmetric storage, in the
// step's tile layout: slot = pixel, chunk = 4 of the 81 offsets in scanline
// order (0 where the neighbour or the pixel is outside the patch, and 3 zeros
// at the end).  A thread owns a slot, so a warp's 16-byte stores of a chunk
// are 512 contiguous bytes; its pixels are 2 tile rows, so the plane reads
// stay coalesced.
__global__ void __launch_bounds__(kTilePx) cf_full(const PatchDev* __restrict__ patches,
                                                   const int4* __restrict__ work, const float* __restrict__ a_up,
                                                   const float* __restrict__ a_diag, long long lvec,
                                                   float* __restrict__ afull) {
  constexpr int NCH = DiskStencil::NC / 4, ctr = kStencilN / 2;
  const int4 w = work[blockIdx.x];
  const PatchDev P = patches[w.x];
  const int t = threadIdx.x, k = (t >> 2) & 7;
  const int y = w.y + 2 * (t >> 5) + (k >> 2), x = w.z + 4 * (t & 3) + (k & 3);
  const bool inside = y < P.H && x < P.W;
  const long long p = P.vec + (long long)y * P.W + x;
  float4* dst = (float4*)afull + (long long)blockIdx.x * NCH * kTilePx + t;
#pragma unroll 3
  for (int e4 = 0; e4 < NCH; e4++) {
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int e = 4 * e4 + j;
      v[j] = 0.f;
      if (e >= kStencilN || !inside) continue;
      if (e == ctr) {
        v[j] = a_diag[p];
        continue;
      }
      // upper offsets are c_bup[e - 41]; the disk is point-symmetric, so
      // lower offset e mirrors upper offset 80 - e
      const int u = e > ctr ? e - ctr - 1 : kStencilN - 1 - e - ctr - 1;
      const int dy = e > ctr ? c_bup_dy[u] : -c_bup_dy[u];
      const int dx = e > ctr ? c_bup_dx[u] : -c_bup_dx[u];
      const int yy = y + dy, xx = x + dx;
      if (yy >= 0 && yy < P.H && xx >= 0 && xx < P.W)
        v[j] = e > ctr ? a_up[(long long)u * lvec + p] : a_up[(long long)u * lvec + p + (long long)dy * P.W + dx];
    }
    dst[(long long)e4 * kTilePx] = make_float4(v[0], v[1], v[2], v[3]);
  }
}

// ------------------------------------------------------------------ Gram
__device__ __forceinline__ void ffp(float& hi, float& lo, float a, float b) {
  // __fmul_rn / __fadd_rn: never contracted into an FMA, which would break
  // the error-free transformations
  const float p = __fmul_rn(a, b);
  const float pe = fmaf(a, b, -p);
  const float s = __fadd_rn(hi, p);
  const float z = s - hi;
  lo += ((hi - (s - z)) + (p - z)) + pe;
  hi = s;
}

// G = U^T V over a tile of pixels.  Chunks of 256 pixel rows of U and V are
// staged in shared memory; four groups of 64 threads take 64 rows each, a
// thread owning a 4 x 4 block of G (two broadcast 16-byte loads feed 16
// FMAs).  Each group's 64-term FP32 FMA runs are folded into a float-float
// (hi, lo) pair by an error-free TwoSum, so the sum over the tile is as
// accurate as a compensated one at about the cost of plain FMAs; the four
// groups and then the tiles are summed in FP64.
constexpr int GR_CH = 256;  // pixels per staged chunk
__device__ __forceinline__ void two_sum_into(F2& hi, F2& lo, F2 x) {
  const F2 s = f2_add(hi, x);
  const F2 bb = f2_sub(s, hi);
  lo = f2_add(lo, f2_add(f2_sub(hi, f2_sub(s, bb)), f2_sub(x, bb)));
  hi = s;
}

// The reductions and the rotation split each eigensolver tile (kEigTile
// pixels) into kBlkSplit runs, one CTA each, so a launch has several CTAs
// per SM and no near-empty last wave.  A CTA's partial sums are float-float
// pairs in slot blockIdx.x of a.part; the slots [tile_begin, tile_begin +
// tile_count) x kBlkSplit of a patch are added in order, in float-float on the
// FP32 pipes (FP64 would take tens of microseconds at GB300's rate): by
// cf_gram_sum, or for cf_resid by the patch's last CTA.
__device__ __forceinline__ void ff2_add(float2& s, float2 b) {
  const float t = s.x + b.x;
  const float z = t - s.x;
  s.y += ((s.x - (t - z)) + (b.x - z)) + b.y;
  s.x = t;
}
struct BlkRun {
  EigTile t;
  int p0, p1;
};
__device__ __forceinline__ BlkRun blk_run(const BlkArgs& a) {
  BlkRun r;
  r.t = a.tiles[blockIdx.x / kBlkSplit];
  const int len = (r.t.p1 - r.t.p0 + kBlkSplit - 1) / kBlkSplit;
  r.p0 = min(r.t.p1, r.t.p0 + (int)(blockIdx.x % kBlkSplit) * len);
  r.p1 = min(r.t.p1, r.p0 + len);
  return r;
}
// true in every thread of the last CTA of patch t.patch to arrive
__device__ __forceinline__ bool blk_last(const BlkArgs& a, int patch) {
  __shared__ int is_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const int prev = atomicAdd(a.counter + patch, 1);
    is_last = (prev == a.tile_count[patch] * kBlkSplit - 1);
    if (is_last) a.counter[patch] = 0;
  }
  __syncthreads();
  if (is_last) __threadfence();
  return is_last;
}
// sum of element e over the patch's CTA slots (stride floats2 per slot), in
// order; the loads of 32 slots are in flight together
__device__ __forceinline__ double blk_sum(const BlkArgs& a, int patch, int e, int stride) {
  constexpr int NB = 32;
  const int b0 = a.tile_begin[patch] * kBlkSplit, b1 = b0 + a.tile_count[patch] * kBlkSplit;
  const float2* part = (const float2*)a.part + (long long)b0 * stride + e;
  float2 acc = make_float2(0.f, 0.f);
  for (int b = b0; b < b1; b += NB, part += (long long)NB * stride) {
    float2 v[NB];
#pragma unroll
    for (int i = 0; i < NB; i++) v[i] = b + i < b1 ? part[(long long)i * stride] : make_float2(0.f, 0.f);
#pragma unroll
    for (int i = 0; i < NB; i++) ff2_add(acc, v[i]);  // a pair of zeros changes nothing
  }
  return (double)acc.x + (double)acc.y;
}

// TWO: one pass computes out = U^T V and out2 = U^T U (the Rayleigh-Ritz
// step's two Gram matrices), each element with the same operations in the
// same order as a pass of its own, so the results are the same to the bit.
template <bool TWO>
__global__ void __launch_bounds__(256, TWO ? 2 : 3) cf_gram(BlkArgs a, const float* __restrict__ U,
                                                            const float* __restrict__ V) {
  const BlkRun run = blk_run(a);
  const EigTile t = run.t;
  if (!a.active[t.patch]) return;
  const PatchDev P = a.patches[t.patch];
  extern __shared__ __align__(16) float gsm[];  // us[GR_CH][32], vs[GR_CH][32]; reused for the group sums
  float* us = gsm;
  float* vs = gsm + GR_CH * kBlk;
  const int grp = threadIdx.x >> 6, lt = threadIdx.x & 63;
  const int i0 = (lt >> 3) * 4, j0 = (lt & 7) * 4;
  constexpr int NG = TWO ? 2 : 1;  // Gram matrices formed
  F2 hi[NG][8], lo[NG][8];         // pairs of columns: [row of the 4 x 4 block][pair]
#pragma unroll
  for (int g = 0; g < NG; g++)
#pragma unroll
    for (int k = 0; k < 8; k++) hi[g][k] = lo[g][k] = f2(0.f, 0.f);
  for (int p0 = run.p0; p0 < run.p1; p0 += GR_CH) {
    __syncthreads();
    for (int f = threadIdx.x; f < GR_CH * kBlk / 4; f += blockDim.x) {
      const int pp = f / (kBlk / 4), c4 = f % (kBlk / 4);
      const int p = p0 + pp;
      float4 u = make_float4(0.f, 0.f, 0.f, 0.f), v = u;
      if (p < run.p1) {
        u = ((const float4*)(U + (P.vec + p) * kBlk))[c4];
        v = ((const float4*)(V + (P.vec + p) * kBlk))[c4];
      }
      ((float4*)us)[f] = u;
      ((float4*)vs)[f] = v;
    }
    __syncthreads();
    F2 acc[NG][8];
#pragma unroll
    for (int g = 0; g < NG; g++)
#pragma unroll
      for (int k = 0; k < 8; k++) acc[g][k] = f2(0.f, 0.f);
    const int pbeg = grp * (GR_CH / 4);
#pragma unroll(TWO ? 2 : 4)
    for (int pp = pbeg; pp < pbeg + GR_CH / 4; pp++) {
      const float4 u4 = *(const float4*)(us + pp * kBlk + i0);
      const float4 v4 = *(const float4*)(vs + pp * kBlk + j0);
      const F2 uu[4] = {f2(u4.x, u4.x), f2(u4.y, u4.y), f2(u4.z, u4.z), f2(u4.w, u4.w)};
      const F2 vv[2] = {f2(v4.x, v4.y), f2(v4.z, v4.w)};
#pragma unroll
      for (int r = 0; r < 4; r++)
#pragma unroll
        for (int c = 0; c < 2; c++) acc[0][r * 2 + c] = f2_fma(uu[r], vv[c], acc[0][r * 2 + c]);
      if constexpr (TWO) {
        const float4 w4 = *(const float4*)(us + pp * kBlk + j0);
        const F2 ww[2] = {f2(w4.x, w4.y), f2(w4.z, w4.w)};
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
          for (int c = 0; c < 2; c++) acc[NG - 1][r * 2 + c] = f2_fma(uu[r], ww[c], acc[NG - 1][r * 2 + c]);
      }
    }
#pragma unroll
    for (int g = 0; g < NG; g++)
#pragma unroll
      for (int k = 0; k < 8; k++) two_sum_into(hi[g][k], lo[g][k], acc[g][k]);
  }
  // the four groups' blocks, summed in float-float
  __syncthreads();
  float2* red = (float2*)gsm;  // [NG][4][32 * 32] (64 KB for two)
#pragma unroll
  for (int g = 0; g < NG; g++)
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const float2 h = f2_split(hi[g][k]), l = f2_split(lo[g][k]);
      float2* at = red + (g * 4 + grp) * kBlk * kBlk + (i0 + k / 2) * kBlk + j0 + 2 * (k % 2);
      at[0] = make_float2(h.x, l.x);
      at[1] = make_float2(h.y, l.y);
    }
  __syncthreads();
  float2* part = (float2*)a.part + (long long)blockIdx.x * NG * kBlk * kBlk;
  for (int e = threadIdx.x; e < NG * kBlk * kBlk; e += blockDim.x) {
    const int g = e / (kBlk * kBlk), el = e % (kBlk * kBlk);
    float2 sum = red[g * 4 * kBlk * kBlk + el];
    for (int q = 1; q < 4; q++) ff2_add(sum, red[(g * 4 + q) * kBlk * kBlk + el]);
    part[e] = sum;
  }
}

// The Gram matrices' sums over a patch's CTA slots, 128 elements per CTA: a
// patch of 0.4 Mpx has 800 slots (13 MB for two matrices), which its last
// cf_gram CTA alone took longer to add than the others to form.  It pays for
// few slots too: cf_gram + this launch take 8.6 + 2.5 us for one matrix of a
// 64 x 80 image (12 slots) and 12.2 + 2.5 for two, from 13.4 and 20.0 us with
// the last CTA adding; 9.4 + 6.7 from 30.1 and 13.0 + 6.7 from 52.8 for 266^2.
constexpr int kSumThreads = 128;
__global__ void __launch_bounds__(kSumThreads) cf_gram_sum(BlkArgs a, int ngram, double* __restrict__ out,
                                                           double* __restrict__ out2) {
  const int patch = blockIdx.x, e = blockIdx.y * kSumThreads + threadIdx.x;
  if (!a.active[patch]) return;
  const int g = e / (kBlk * kBlk), el = e % (kBlk * kBlk);
  (g ? out2 : out)[(long long)patch * kBlk * kBlk + el] = blk_sum(a, patch, e, ngram * kBlk * kBlk);
}

// U <- U M (and V <- V M if V), M = a.mat[patch] (32 x 32, FP64 on the
// host), two pixel rows per thread.  C (the Rayleigh-Ritz rotation): M is
// split into FP32 hi + lo parts; each output sums its products with hi by
// FMA in groups of four, folded into a float-float by an exact TwoSum, and
// its products with lo by FMA into the low word, so the Ritz vectors carry
// little more than FP32 storage rounding; a plain FP32 sum (enough for the
// orthonormalisation passes, which the next Rayleigh-Ritz step corrects)
// leaves ~3e-7 relative error per element.
// Each warp stages its own 64 rows in shared memory -- coalesced 16-byte
// loads in, the rotation on each lane's two rows there, coalesced stores
// out -- synchronising only with __syncwarp, so the warps of a CTA overlap
// their load, compute and store phases.  (Threads loading their own 128-byte
// rows from global memory made every warp access touch 32 lines; staging
// behind CTA-wide barriers serialised the phases.)  Row pitch 36 floats: the
// 8 lanes of a 16-byte access phase reach 8 rows in distinct banks.
constexpr int RW_ROWS = 64, RW_PITCH = kBlk + 4;
constexpr int kRotSmem = 8 * RW_ROWS * RW_PITCH * sizeof(float);
static_assert(8 * RW_ROWS == kEigTile / kBlkSplit, "8 warps x 64 rows cover a CTA's run");
template <bool C>
__global__ void __launch_bounds__(256) cf_rotate(BlkArgs a, float* __restrict__ U, float* __restrict__ V,
                                                 int ncols) {
  const BlkRun run = blk_run(a);
  const EigTile t = run.t;
  if (!a.active[t.patch]) return;
  const PatchDev P = a.patches[t.patch];
  extern __shared__ __align__(16) float rsm[];  // [8 warps][RW_ROWS][RW_PITCH]
  __shared__ __align__(16) float mh[kBlk][kBlk], ml[kBlk][kBlk];
  const double* M = a.mat + (long long)t.patch * kBlk * kBlk;
  for (int e = threadIdx.x; e < kBlk * kBlk; e += blockDim.x) {
    const double m = M[e];
    const float h = (float)m;
    mh[e / kBlk][e % kBlk] = h;
    ml[e / kBlk][e % kBlk] = (float)(m - (double)h);
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wp0 = run.p0 + warp * RW_ROWS;
  const int n = max(0, min(RW_ROWS, run.p1 - wp0));
  float* ws = rsm + warp * RW_ROWS * RW_PITCH;
  for (int which = 0; which < (V ? 2 : 1); which++) {
    float4* g4 = (float4*)((which ? V : U) + (P.vec + wp0) * kBlk);
    for (int f = lane; f < n * (kBlk / 4); f += 32) *(float4*)(ws + (f >> 3) * RW_PITCH + (f & 7) * 4) = g4[f];
    __syncwarp();
    // two rows per lane, so each broadcast load of M feeds both
    if (lane < n) {
      const bool ok1 = lane + 32 < n;
      float* rows[2];
      rows[0] = ws + lane * RW_PITCH;
      rows[1] = ok1 ? rows[0] + 32 * RW_PITCH : rows[0];
      float x[2][kBlk];
#pragma unroll
      for (int k = 0; k < 2; k++)
#pragma unroll
        for (int c = 0; c < kBlk; c += 4) {
          const float4 v = *(const float4*)(rows[k] + c);
          x[k][c] = v.x;
          x[k][c + 1] = v.y;
          x[k][c + 2] = v.z;
          x[k][c + 3] = v.w;
        }
#pragma unroll 1
      for (int c0 = 0; c0 < kBlk; c0 += 4) {
        F2 hi[2][2], lo[2][2], g[2][2];  // pairs of columns
#pragma unroll
        for (int k = 0; k < 2; k++)
#pragma unroll
          for (int j = 0; j < 2; j++) hi[k][j] = lo[k][j] = g[k][j] = f2(0.f, 0.f);
#pragma unroll
        for (int r = 0; r < kBlk; r++) {
          const float4 h4 = *(const float4*)&mh[r][c0];  // broadcast: every thread reads the same row
          const F2 hh[2] = {f2(h4.x, h4.y), f2(h4.z, h4.w)};
          F2 ll[2] = {f2(0.f, 0.f), f2(0.f, 0.f)};
          if constexpr (C) {
            const float4 l4 = *(const float4*)&ml[r][c0];
            ll[0] = f2(l4.x, l4.y);
            ll[1] = f2(l4.z, l4.w);
          }
#pragma unroll
          for (int k = 0; k < 2; k++) {
            const F2 xr = f2(x[k][r], x[k][r]);
#pragma unroll
            for (int j = 0; j < 2; j++) {
              if constexpr (C) {
                g[k][j] = f2_fma(xr, hh[j], g[k][j]);
                lo[k][j] = f2_fma(xr, ll[j], lo[k][j]);
                if ((r & 3) == 3) {  // r is a compile-time constant here
                  const F2 sum = f2_add(hi[k][j], g[k][j]), z = f2_sub(sum, hi[k][j]);
                  lo[k][j] = f2_add(lo[k][j], f2_add(f2_sub(hi[k][j], f2_sub(sum, z)), f2_sub(g[k][j], z)));
                  hi[k][j] = sum;
                  g[k][j] = f2(0.f, 0.f);
                }
              } else {
                hi[k][j] = f2_fma(xr, hh[j], hi[k][j]);
              }
            }
          }
        }
        if (c0 < ncols) {
#pragma unroll
          for (int k = 0; k < 2; k++) {
            if (k && !ok1) break;
            const float2 a0 = f2_split(f2_add(hi[k][0], lo[k][0])), a1 = f2_split(f2_add(hi[k][1], lo[k][1]));
            *(float4*)(rows[k] + c0) = make_float4(a0.x, a0.y, a1.x, a1.y);
          }
        }
      }
    }
    __syncwarp();
    for (int f = lane; f < n * (kBlk / 4); f += 32) g4[f] = *(const float4*)(ws + (f >> 3) * RW_PITCH + (f & 7) * 4);
    __syncwarp();
  }
}

// per-column |A x_c - theta_c x_c|^2 (AX and X given), last CTA sums
__global__ void __launch_bounds__(256) cf_resid(BlkArgs a, const float* __restrict__ X,
                                                const float* __restrict__ AX, double* __restrict__ out) {
  const BlkRun run = blk_run(a);
  const EigTile t = run.t;
  if (!a.active[t.patch]) return;
  const PatchDev P = a.patches[t.patch];
  const int c = threadIdx.x & 31, lanegroup = threadIdx.x >> 5;
  const float th = (float)a.theta[(long long)t.patch * kBlk + c];
  float hi = 0.f, lo = 0.f;
#pragma unroll 4
  for (int p = run.p0 + lanegroup; p < run.p1; p += 8) {
    const long long q = (P.vec + p) * kBlk + c;
    const float r = fmaf(-th, X[q], AX[q]);
    ffp(hi, lo, r, r);
  }
  __shared__ float2 red[8][kBlk];
  red[lanegroup][c] = make_float2(hi, lo);
  __syncthreads();
  if (threadIdx.x < kBlk) {
    float2 sum = red[0][threadIdx.x];
    for (int g = 1; g < 8; g++) ff2_add(sum, red[g][threadIdx.x]);
    ((float2*)a.part)[(long long)blockIdx.x * kBlk + threadIdx.x] = sum;
  }
  if (!blk_last(a, t.patch)) return;
  if (threadIdx.x < kBlk) out[(long long)t.patch * kBlk + threadIdx.x] = blk_sum(a, t.patch, threadIdx.x, kBlk);
}

// columns 0..nvec-1 of X into separate vectors evec[c][vec layout]
__global__ void __launch_bounds__(256) cf_extract(BlkArgs a, const float* __restrict__ X,
                                                  float* __restrict__ evec, int nvec) {
  const EigTile t = a.tiles[blockIdx.x];
  if (!a.done[t.patch]) return;
  const PatchDev P = a.patches[t.patch];
  for (int p = t.p0 + threadIdx.x; p < t.p1; p += blockDim.x)
    for (int c = 0; c < nvec; c++) evec[(long long)c * a.lvec + P.vec + p] = X[(P.vec + p) * kBlk + c];
}

// seeded start block (a fixed hash per pixel and column)
__global__ void __launch_bounds__(256) cf_init(BlkArgs a, float* __restrict__ X) {
  const EigTile t = a.tiles[blockIdx.x];
  if (!a.active[t.patch]) return;
  const PatchDev P = a.patches[t.patch];
  for (int idx = threadIdx.x; idx < (t.p1 - t.p0) * kBlk; idx += blockDim.x) {
    const int p = t.p0 + idx / kBlk, c = idx % kBlk;
    uint32_t x = (uint32_t)p * 2654435761u ^ ((uint32_t)c * 0x9e3779b9u + 0x1234567u);
    x ^= x >> 16;
    x *= 0x7feb352dU;
    x ^= x >> 15;
    x *= 0x846ca68bU;
    x ^= x >> 16;
    X[(P.vec + p) * kBlk + c] = (float)(x & 0xffffff) * (1.0f / 16777216.0f) - 0.5f;
  }
}

// ------------------------------------------------------------ coarse level
// Galerkin coarsening by 2 x 2 aggregation: W_c(P,Q) = sum of W(p,q) over
// p in P, q in Q, so (D_c - W_c) u = lambda D_c u is the projection of the
// fine generalised problem onto block-constant vectors.  Fine radius 5 gives
// coarse offsets up to 3: a full 7 x 7 stencil, stored per offset.
// coarse degrees d_c(P) = the sum of the fine degrees of P's pixels (the
// row sums of W_c, since W_c(P, Q) sums W over P x Q), and D_c^-1/2
__global__ void __launch_bounds__(256) cf_coarse_deg(CoarseArgs c) {
  const int4 w = c.work[blockIdx.x];  // coarse (patch, Y0, X0)
  const PatchDev F = c.fine[w.x], C = c.coarse[w.x];
  const int Y = w.y + threadIdx.x / 16, X = w.z + threadIdx.x % 16;
  if (Y >= C.H || X >= C.W) return;
  double deg = 0.0;
  for (int sy = 0; sy < 2; sy++)
    for (int sx = 0; sx < 2; sx++) {
      const int y = 2 * Y + sy, x = 2 * X + sx;
      if (y < F.H && x < F.W) deg += c.deg[F.vec + (long long)y * F.W + x];
    }
  const long long P = C.vec + (long long)Y * C.W + X;
  c.degc[P] = (float)deg;
  c.disc[P] = (float)(1.0 / sqrt(deg));
}

// coarse stencil index of fine displacement (a, b) from sub-pixel (0, 0):
// coarse offset (floor(a / 2), floor(b / 2)), a, b in [-5, 6]
__host__ __device__ constexpr int cidx(int a, int b) {
  return ((a + 8) / 2 - 4 + kCR) * kCW + (b + 8) / 2 - 4 + kCR;
}
static_assert(cidx(0, 0) == kCR * kCW + kCR && cidx(-5, -5) == 0 && cidx(6, 6) == kCN - 1, "coarse offsets");

// upper offset j's displacement (the inverse of upper_k)
__host__ __device__ constexpr int upper_dy_from(int j, int dy) {
  return j < 2 * disk_half_width(dy) + 1 ? dy : upper_dy_from(j - 2 * disk_half_width(dy) - 1, dy + 1);
}
__host__ __device__ constexpr int upper_dy(int j) { return j < kStencilR ? 0 : upper_dy_from(j - kStencilR, 1); }
__host__ __device__ constexpr int upper_dx(int j) {
  return upper_dy(j) == 0 ? j + 1 : j - upper_k(upper_dy(j), 0);
}
static_assert(upper_dy(0) == 0 && upper_dx(0) == 1 && upper_dy(5) == 1 && upper_dx(5) == -4 &&
                  upper_dy(kUpper - 1) == kStencilR && upper_dx(kUpper - 1) == 0 && upper_k(upper_dy(23), upper_dx(23)) == 23,
              "upper offset inverse");

// the terms of fine sub-pixel (SY, SX) of a coarse pixel: upper offset J's
// lower neighbour q = p - (dy,dx) (its upper entry at q), then its upper
// neighbour q = p + (dy,dx); each lands on a compile-time coarse offset
template <int SY, int SX, int J>
__device__ __forceinline__ void coarsen_terms(float (&acc)[kCN], const float* __restrict__ wsym, long long lvec,
                                              long long p, int y, int x, int H, int W) {
  if constexpr (J < kUpper) {
    constexpr int dy = upper_dy(J), dx = upper_dx(J);
    const float* plane = wsym + (long long)J * lvec;
    if (y - dy >= 0 && x - dx >= 0 && x - dx < W) acc[cidx(SY - dy, SX - dx)] += plane[p - (dy * W + dx)];
    if (y + dy < H && x + dx >= 0 && x + dx < W) acc[cidx(SY + dy, SX + dx)] += plane[p];
    coarsen_terms<SY, SX, J + 1>(acc, wsym, lvec, p, y, x, H, W);
  }
}
template <int SY, int SX>
__device__ __forceinline__ void coarsen_sub(float (&acc)[kCN], const CoarseArgs& c, const PatchDev& F, int Y, int X) {
  const int y = 2 * Y + SY, x = 2 * X + SX;
  if (y < F.H && x < F.W) {
    acc[kCR * kCW + kCR] += 1.f;  // w_pp = 1
    coarsen_terms<SY, SX, 0>(acc, c.wsym_up, c.lvec_f, F.vec + (long long)y * F.W + x, y, x, F.H, F.W);
  }
}

// W_c row of one coarse pixel, then A_c = I - D_c^-1/2 W_c D_c^-1/2 on it.
// The fine offsets, the two signs and the 2 x 2 sub-pixels are unrolled at
// compile time, so every term's coarse offset -- floor((s + dy) / 2) for
// sub-pixel s -- is a constant and the 49 sums stay in registers.  Terms
// are added per sum in the order: sub-pixel, upper offset, lower before
// upper neighbour.
// The rows go out in the step's tile layout (see cf_full).
__global__ void __launch_bounds__(kTilePx) cf_coarsen(CoarseArgs c) {
  const int4 w = c.work[blockIdx.x];
  const PatchDev F = c.fine[w.x], C = c.coarse[w.x];
  constexpr int NCH = SquareStencil::NC / 4;
  const int t = threadIdx.x, pk = (t >> 2) & 7;
  const int Y = w.y + 2 * (t >> 5) + (pk >> 2), X = w.z + 4 * (t & 3) + (pk & 3);
  const bool inside = Y < C.H && X < C.W;
  float acc[kCN];
#pragma unroll
  for (int k = 0; k < kCN; k++) acc[k] = 0.f;
  float dp = 0.f;
  const long long P = C.vec + (long long)Y * C.W + X;
  if (inside) {
    coarsen_sub<0, 0>(acc, c, F, Y, X);
    coarsen_sub<0, 1>(acc, c, F, Y, X);
    coarsen_sub<1, 0>(acc, c, F, Y, X);
    coarsen_sub<1, 1>(acc, c, F, Y, X);
    dp = c.disc[P];
  }
  float4* dst = (float4*)c.wc + (long long)blockIdx.x * NCH * kTilePx + t;
#pragma unroll
  for (int q = 0; q < NCH; q++) {
    float v[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int k = 4 * q + j;
      v[j] = 0.f;
      if (k >= kCN || !inside) continue;
      const int dY = k / kCW - kCR, dX = k % kCW - kCR;
      const int YY = Y + dY, XX = X + dX;
      if (YY >= 0 && YY < C.H && XX >= 0 && XX < C.W)
        v[j] = -acc[k] * dp * c.disc[C.vec + (long long)YY * C.W + XX];
      if (k == kCR * kCW + kCR) v[j] += 1.f;
    }
    dst[(long long)q * kTilePx] = make_float4(v[0], v[1], v[2], v[3]);
  }
}

// fine start block from the coarse Ritz vectors: the coarse generalised
// eigenvectors u_c = D_c^-1/2 y_c interpolated bilinearly to the fine pixel
// centres (clamped at the patch border), then y = D^1/2 u.  Smoother than
// the piecewise-constant P u_c of the Galerkin pair, so the fine level
// starts closer to its eigenvectors.
__global__ void __launch_bounds__(256) cf_prolong(CoarseArgs c, const float* __restrict__ xc,
                                                  float* __restrict__ xf) {
  const int4 w = c.work_f[blockIdx.x];  // fine (patch, y0, x0)
  const PatchDev F = c.fine[w.x], C = c.coarse[w.x];
  const int y = w.y + threadIdx.x / 16, x = w.z + threadIdx.x % 16;
  if (y >= F.H || x >= F.W) return;
  const long long p = F.vec + (long long)y * F.W + x;
  // fine centre in coarse pixel coordinates
  const float cy = fminf(fmaxf((y + 0.5f) * 0.5f - 0.5f, 0.f), (float)(C.H - 1));
  const float cx = fminf(fmaxf((x + 0.5f) * 0.5f - 0.5f, 0.f), (float)(C.W - 1));
  const int y0 = (int)cy, x0 = (int)cx;
  const int y1 = min(y0 + 1, C.H - 1), x1 = min(x0 + 1, C.W - 1);
  const float fy = cy - y0, fx = cx - x0;
  const long long P00 = C.vec + (long long)y0 * C.W + x0, P01 = C.vec + (long long)y0 * C.W + x1;
  const long long P10 = C.vec + (long long)y1 * C.W + x0, P11 = C.vec + (long long)y1 * C.W + x1;
  const float sq = sqrtf(c.deg[p]);
  const float w00 = (1.f - fy) * (1.f - fx) * c.disc[P00] * sq, w01 = (1.f - fy) * fx * c.disc[P01] * sq;
  const float w10 = fy * (1.f - fx) * c.disc[P10] * sq, w11 = fy * fx * c.disc[P11] * sq;
  const float4* a = (const float4*)(xc + P00 * kBlk);
  const float4* b = (const float4*)(xc + P01 * kBlk);
  const float4* cc = (const float4*)(xc + P10 * kBlk);
  const float4* d = (const float4*)(xc + P11 * kBlk);
  float4* dst = (float4*)(xf + p * kBlk);
#pragma unroll
  for (int c4 = 0; c4 < kBlk / 4; c4++) {
    const float4 va = a[c4], vb = b[c4], vc = cc[c4], vd = d[c4];
    float4 v;
    v.x = w00 * va.x + w01 * vb.x + w10 * vc.x + w11 * vd.x;
    v.y = w00 * va.y + w01 * vb.y + w10 * vc.y + w11 * vd.y;
    v.z = w00 * va.z + w01 * vb.z + w10 * vc.z + w11 * vd.z;
    v.w = w00 * va.w + w01 * vb.w + w10 * vc.w + w11 * vd.w;
    dst[c4] = v;
  }
}

cudaError_t cf_launch_coarsen(const CoarseArgs& c, int nwork_c, cudaStream_t s) {
  cf_coarse_deg<<<nwork_c, 256, 0, s>>>(c);
  cf_coarsen<<<nwork_c, kTilePx, 0, s>>>(c);
  return cudaGetLastError();
}
cudaError_t cf_launch_prolong(const CoarseArgs& c, int nwork_f, const float* xc, float* xf, cudaStream_t s) {
  cf_prolong<<<nwork_f, 256, 0, s>>>(c, xc, xf);
  return cudaGetLastError();
}

template <class S, bool C, int SBR>
static cudaError_t step_go(const BlkArgs& a, const int4* work, int nwork, const float* Y, const float* X, float* out,
                           int step, int nsm, bool overlap, cudaStream_t s) {
  using SM = StepSmem<S, kStepWarps, SBR>;
  static PerDevice ready;
  const cudaError_t e = ready.once([] { return grant_smem(cf_step_t<S, C, kStepWarps, SBR>, SM::bytes); });
  if (e != cudaSuccess) return e;
  // one persistent CTA per SM
  return launch_overlap(cf_step_t<S, C, kStepWarps, SBR>, std::min(nwork * (kStepTile / SM::ROWS), nsm),
                        (kStepWarps + 2) * 32, SM::bytes, s, overlap, a, work, nwork, Y, X, out, step);
}
template <class S, bool C>
static cudaError_t step_go(const BlkArgs& a, const int4* work, int nwork, const float* Y, const float* X, float* out,
                           int step, int nsm, int variant, bool overlap, cudaStream_t s) {
  return variant == 0 ? step_go<S, C, 2>(a, work, nwork, Y, X, out, step, nsm, overlap, s)
                      : step_go<S, C, 1>(a, work, nwork, Y, X, out, step, nsm, overlap, s);
}

cudaError_t cf_launch_step(const BlkArgs& a, const int4* work, int nwork, const float* Y, const float* X, float* out,
                           int step, cudaStream_t s, bool comp, int variant, bool overlap) {
  if (nwork <= 0) return cudaSuccess;
  int dev = 0, nsm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  if (a.coarse)
    e = comp ? step_go<SquareStencil, true>(a, work, nwork, Y, X, out, step, nsm, variant, overlap, s)
             : step_go<SquareStencil, false>(a, work, nwork, Y, X, out, step, nsm, variant, overlap, s);
  else
    e = comp ? step_go<DiskStencil, true>(a, work, nwork, Y, X, out, step, nsm, variant, overlap, s)
             : step_go<DiskStencil, false>(a, work, nwork, Y, X, out, step, nsm, variant, overlap, s);
  return e != cudaSuccess ? e : cudaGetLastError();
}
cudaError_t cf_launch_full(const PatchDev* patches, const int4* work16, int nwork, const float* a_up,
                           const float* a_diag, long long lvec, float* afull, cudaStream_t s) {
  cf_full<<<nwork, kTilePx, 0, s>>>(patches, work16, a_up, a_diag, lvec, afull);
  return cudaGetLastError();
}
cudaError_t cf_launch_gram(const BlkArgs& a, int npatch, int ntiles, const float* U, const float* V, double* out,
                           cudaStream_t s, double* out2) {
  constexpr int smem = 2 * GR_CH * kBlk * sizeof(float);  // 64 KB; the group sums (32 or 64 KB) reuse it
  static PerDevice ready;
  const cudaError_t e = ready.once([] {
    const cudaError_t f = grant_smem(cf_gram<false>, smem);
    return f != cudaSuccess ? f : grant_smem(cf_gram<true>, smem);
  });
  if (e != cudaSuccess) return e;
  if (out2)
    cf_gram<true><<<ntiles * kBlkSplit, 256, smem, s>>>(a, U, V);
  else
    cf_gram<false><<<ntiles * kBlkSplit, 256, smem, s>>>(a, U, V);
  const int ngram = out2 ? 2 : 1;
  cf_gram_sum<<<dim3(npatch, ngram * kBlk * kBlk / kSumThreads), kSumThreads, 0, s>>>(a, ngram, out, out2);
  return cudaGetLastError();
}
cudaError_t cf_launch_rotate(const BlkArgs& a, int ntiles, float* U, float* V, int ncols, cudaStream_t s,
                             bool comp) {
  static PerDevice ready;
  const cudaError_t e = ready.once([] {
    const cudaError_t f = grant_smem(cf_rotate<false>, kRotSmem);
    return f != cudaSuccess ? f : grant_smem(cf_rotate<true>, kRotSmem);
  });
  if (e != cudaSuccess) return e;
  if (comp)
    cf_rotate<true><<<ntiles * kBlkSplit, 256, kRotSmem, s>>>(a, U, V, ncols);
  else
    cf_rotate<false><<<ntiles * kBlkSplit, 256, kRotSmem, s>>>(a, U, V, ncols);
  return cudaGetLastError();
}
cudaError_t cf_launch_resid(const BlkArgs& a, int ntiles, const float* X, const float* AX, double* out,
                            cudaStream_t s) {
  cf_resid<<<ntiles * kBlkSplit, 256, 0, s>>>(a, X, AX, out);
  return cudaGetLastError();
}
cudaError_t cf_launch_extract(const BlkArgs& a, int ntiles, const float* X, float* evec, int nvec,
                              cudaStream_t s) {
  cf_extract<<<ntiles, 256, 0, s>>>(a, X, evec, nvec);
  return cudaGetLastError();
}
cudaError_t cf_launch_init(const BlkArgs& a, int ntiles, float* X, cudaStream_t s) {
  cf_init<<<ntiles, 256, 0, s>>>(a, X);
  return cudaGetLastError();
}

}  // namespace gpb
