// k_cues.cu -- oriented half-disc histogram gradients, mPb combination and
// oriented non-maximum suppression (sm_103a).
//
// Reference: lib_image::hist_gradient_2D / compute_hist_gradient_2D
// (globalPb/src/math/libraries/lib_image.cc:3120-3235, 3575-3686) as called by
// mex_pb_parts_final_selected.cpp:157-227, the weighted sum of
// multiscalePb.cpp:217-245 and nonmax_channels + nonmax_oriented_2D
// (src/nonmax_channels.cpp:8-80, lib_image.cc:4083-4197).
//
// One warp computes one pixel.  The four label images (L, a, b bins and the
// texton) are packed into one u32 per pixel and staged, reflect-padded by 20,
// in shared memory.  The radius-20 disc is walked in four nested annuli
// (r <= 3, 5, 10, 20); slice membership does not depend on r, so the counts
// are cumulative and one walk serves every (cue, radius) pair.  Lane
// l = half*16 + slice owns one byte per cue and bin, so no atomics are
// needed.  After each annulus the lanes switch role, first to histogram bins
// (slice masses, normalisation, the 8-step spin), then to (8 bins,
// orientation) pairs for the Gaussian bin smoothing and the chi-squared
// terms.  Smoothing is linear and applied after the per-slice scaling, so 9
// convolutions (the half-disc total and 8 left-right differences) replace
// the 16 per-slice ones.
//
// Measured on 16 patches of 266^2 (1.11 Mpx): 6.9 ms, from 14.2 ms with a
// lane per bin throughout (every smoothing tap loaded 9 shared values for 9
// FMAs, every lane formed all 16 reciprocals, counts were read byte by byte);
// the results are the same to the bit.
#include <float.h>
#include <stdint.h>

#include "gpb_internal.h"
#include "kernels.h"
#include "per_device.h"

namespace gpb {

constexpr int kAnnMax = 1400;
constexpr int kAnnRows = 48;  // rows of the lane-interleaved disc offsets
__constant__ int16_t c_ann_dy[kAnnMax];
__constant__ int16_t c_ann_dx[kAnnMax];
__constant__ int c_ann_start[kNannulus][32];
__constant__ int c_ann_count[kNannulus][32];
__constant__ int c_ann_row[kNannulus + 1];  // first row of an annulus in the lane-interleaved offsets
__constant__ float c_slice_rcp[kNannulus][16];
__constant__ float c_kbg[17];
__constant__ float c_kcg[9];
__constant__ float c_wm[kNcue], c_wg[kNcue];
__constant__ int c_nms_nb[kNori][4][2];
__constant__ float c_nms_d[kNori];
__constant__ float c_nms_cos[kNori][kNori];

cudaError_t upload_cues(const HostTables& t, cudaStream_t s) {
  int16_t dy[kAnnMax] = {}, dx[kAnnMax] = {};
  const int n = (int)t.ann_dy.size();
  for (int i = 0; i < n && i < kAnnMax; i++) {
    dy[i] = t.ann_dy[i];
    dx[i] = t.ann_dx[i];
  }
  float sr[kNannulus][16];  // 1 / pixels of a slice
  int row[kNannulus + 1] = {};
  for (int a = 0; a < kNannulus; a++) {
    int most = 0;
    for (int q = 0; q < 16; q++) sr[a][q] = t.slice_pixels[a][q] ? 1.0f / (float)t.slice_pixels[a][q] : 0.f;
    for (int l = 0; l < 32; l++) most = t.ann_count[a][l] > most ? t.ann_count[a][l] : most;
    row[a + 1] = row[a] + most;
  }
  if (row[kNannulus] > kAnnRows) return cudaErrorInvalidValue;  // the disc's offsets do not fit
  cudaMemcpyToSymbolAsync(c_ann_dy, dy, sizeof(dy), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_ann_dx, dx, sizeof(dx), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_ann_start, t.ann_start, sizeof(t.ann_start), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_ann_count, t.ann_count, sizeof(t.ann_count), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_ann_row, row, sizeof(row), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_slice_rcp, sr, sizeof(sr), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_kbg, t.kbg, sizeof(t.kbg), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_kcg, t.kcg, sizeof(t.kcg), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_wm, t.w_mpb, sizeof(t.w_mpb), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_wg, t.w_g, sizeof(t.w_g), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_nms_nb, t.nms_nb, sizeof(t.nms_nb), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_nms_d, t.nms_d, sizeof(t.nms_d), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_nms_cos, t.nms_cos, sizeof(t.nms_cos), 0, cudaMemcpyHostToDevice, s);
  return cudaSuccess;
}

__device__ __forceinline__ int reflect_c(int i, int n) {
  for (int it = 0; it < 4 && (i < 0 || i >= n); it++) i = (i < 0) ? -i - 1 : 2 * n - 1 - i;
  return i < 0 ? 0 : (i >= n ? n - 1 : i);
}

constexpr unsigned FULL = 0xffffffffu;
constexpr int CT_H = kCueTileH, CT_W = kCueTileW;
constexpr int CT_PH = CT_H + 2 * kMaxRadius, CT_PW = CT_W + 2 * kMaxRadius;
constexpr int CT_WARPS = CT_H;              // one warp per tile row
constexpr int kLabBins = 25;                // quantised L, a, b labels (0..24)

// Shared memory of one warp.  Counters: per cue and bin 32 one-byte counts,
// one per (half, slice) row, at a 48-byte pitch, so lane = bin reads its 32
// counts with two conflict-free 16-byte loads and lane = row increments its
// own byte.  Rows of the bin smoothing: [8 orientation differences, total]
// [8 zeros | 32 bins | 8 zeros], pitch 52 floats, so the 16-byte window loads
// of 8 orientations reach distinct banks and taps outside [0, 32) read 0.
constexpr int HPITCH = 48;
constexpr int HCUE = kLabBins * HPITCH;     // bytes of one colour cue's counters
constexpr int HWARP = 3 * HCUE + kMaxBins * HPITCH;
constexpr int DPITCH = 52, DPAD = 8;
constexpr int DWARP = 9 * DPITCH + kMaxBins + 16;  // rows, 1 / total per bin, 1 / mass per slice
constexpr int CT_OFFS = CT_PH * CT_PW * 4;
constexpr int CT_HIST = CT_OFFS + kAnnRows * 32 * 2;
constexpr int CT_ROWS = CT_HIST + CT_WARPS * HWARP;
constexpr size_t kCueSmem = (size_t)CT_ROWS + (size_t)CT_WARPS * DWARP * 4;
static_assert(HCUE % 16 == 0 && HWARP % 16 == 0 && CT_HIST % 16 == 0 && (DWARP * 4) % 16 == 0, "alignment");
static_assert(DPITCH % 8 == 4 && DPITCH >= DPAD + kMaxBins + DPAD, "smoothing rows");

// Sum of 16 per-lane values over the warp, for all 16 at once: each exchange
// step halves the number of live values (8+4+2+1+1 shuffles).  Lane l returns
// the total of index l >> 1.
__device__ __forceinline__ float warp_sum16(float (&v)[16], int lane) {
  const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4, b1 = lane & 2;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const float keep = b4 ? v[i + 8] : v[i], give = b4 ? v[i] : v[i + 8];
    v[i] = keep + __shfl_xor_sync(FULL, give, 16);
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float keep = b3 ? v[i + 4] : v[i], give = b3 ? v[i] : v[i + 4];
    v[i] = keep + __shfl_xor_sync(FULL, give, 8);
  }
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const float keep = b2 ? v[i + 2] : v[i], give = b2 ? v[i] : v[i + 2];
    v[i] = keep + __shfl_xor_sync(FULL, give, 4);
  }
  {
    const float keep = b1 ? v[1] : v[0], give = b1 ? v[0] : v[1];
    v[0] = keep + __shfl_xor_sync(FULL, give, 2);
  }
  return v[0] + __shfl_xor_sync(FULL, v[0], 1);
}

// the kernel mass that source bin `lane` keeps in range [0, nb) under a
// K-tap bin smoothing; per patch, so computed once per warp
template <int K>
__device__ __forceinline__ float bin_mass(const float* kern, int lane, int nb) {
  float m = 0.f;
#pragma unroll
  for (int j = 0; j < K; j++) {
    const int n = lane + j - K / 2;
    if (n >= 0 && n < nb) m += kern[j];
  }
  return m;
}

__device__ __forceinline__ void unpack16(const uint4& w, float (&f)[16]) {
  const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int q = 0; q < 16; q++) f[q] = (float)((u[q >> 2] >> (8 * (q & 3))) & 255u);
}

// One (cue, radius): the counts of the 16 slices -> the chi-squared terms of
// 8 orientations and all bins, accumulated with the two weight sets.
//   lane = bin      counts, slice masses, normalised differences D_o and
//                   total T, the smoothing of T and its reciprocal
//   lane = (g, o)   o = lane & 7, g = lane >> 3: the smoothing of D_o and the
//                   terms of bins 8 g .. 8 g + 7, from one window of the row
//                   in registers (K + 7 values, 16-byte loads), so a loaded
//                   value feeds up to 8 outputs instead of one
// The truncated 'same' bin convolution (conv_in_place_1D, lib_image.cc:
// 3084-3115) reads zeros outside the 32 bins.  K = 0: no smoothing.
template <int K, bool kRaw>
__device__ __forceinline__ void cue_combo(const uint8_t* cnt, int lane, int nb, int ann, const float* kern, float m,
                                          float wm, float wg, float (&accm)[8], float (&accg)[8], float* raw,
                                          long long raw_stride, float* dsm) {
  constexpr int NB = K > 0 ? kLabBins : kMaxBins;
  float* tsm = dsm + 8 * DPITCH;        // the total's row
  float* rtot = dsm + 9 * DPITCH;       // [32] 1 / smoothed total
  float* rmass = rtot + kMaxBins;       // [16] 1 / slice mass
  uint4 c0 = make_uint4(0u, 0u, 0u, 0u), c1 = c0;
  if (lane < NB) {
    c0 = *(const uint4*)(cnt + lane * HPITCH);
    c1 = *(const uint4*)(cnt + lane * HPITCH + 16);
  }
  // the two halves of a slice: at most 2 x 45 counts, no carry between bytes
  c0.x += c1.x;
  c0.y += c1.y;
  c0.z += c1.z;
  c0.w += c1.w;
  float ch[16];
  unpack16(c0, ch);
  if constexpr (K > 0) {
    float v[16];
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = __fmul_rn(ch[q], m);
    const float S = warp_sum16(v, lane);
    // an empty slice has no counts: any finite factor gives its zeros
    const float r = S != 0.f ? __frcp_rn(S) : 0.f;
    if (!(lane & 1)) rmass[lane >> 1] = r;
    __syncwarp();
#pragma unroll
    for (int q4 = 0; q4 < 4; q4++) {
      const float4 r4 = *(const float4*)(rmass + 4 * q4);
      ch[4 * q4] = __fmul_rn(ch[4 * q4], r4.x);
      ch[4 * q4 + 1] = __fmul_rn(ch[4 * q4 + 1], r4.y);
      ch[4 * q4 + 2] = __fmul_rn(ch[4 * q4 + 2], r4.z);
      ch[4 * q4 + 3] = __fmul_rn(ch[4 * q4 + 3], r4.w);
    }
  } else {
#pragma unroll
    for (int q = 0; q < 16; q++) ch[q] = __fmul_rn(ch[q], c_slice_rcp[ann][q]);
    __syncwarp();  // the rows' previous readers are done
  }
  float T = 0.f, D = 0.f;
#pragma unroll
  for (int q = 0; q < 16; q++) {
    T = __fadd_rn(T, ch[q]);
    D = __fadd_rn(D, q < 8 ? ch[q] : -ch[q]);
  }
#pragma unroll
  for (int o = 0; o < 8; o++) {
    dsm[o * DPITCH + DPAD + lane] = D;
    D = fmaf(2.f, ch[o + 8] - ch[o], D);
  }
  if constexpr (K > 0) tsm[DPAD + lane] = T;
  __syncwarp();
  if constexpr (K > 0) {
    float ct = 0.f;
#pragma unroll
    for (int j = 0; j < K; j++) ct = fmaf(tsm[DPAD + lane + K / 2 - j], kern[j], ct);
    T = ct;
  }
  rtot[lane] = (T != 0.f && lane < nb) ? __frcp_rn(T) : 0.f;
  // this lane's orientation and bins
  const float* row = dsm + (lane & 7) * DPITCH + 8 * (lane >> 3);
  float d[8];
  if constexpr (K > 0) {
    constexpr int R = K / 2, NW = 8 + 2 * R;  // R = 8 or 4: whole 16-byte loads
    float x[NW];
#pragma unroll
    for (int i = 0; i < NW; i += 4) {
      const float4 v = *(const float4*)(row + DPAD - R + i);
      x[i] = v.x;
      x[i + 1] = v.y;
      x[i + 2] = v.z;
      x[i + 3] = v.w;
    }
#pragma unroll
    for (int i = 0; i < 8; i++) d[i] = 0.f;
#pragma unroll
    for (int j = 0; j < K; j++)
#pragma unroll
      for (int i = 0; i < 8; i++) d[i] = fmaf(x[i + 2 * R - j], kern[j], d[i]);
  } else {
#pragma unroll
    for (int i = 0; i < 8; i += 4) {
      const float4 v = *(const float4*)(row + DPAD + i);
      d[i] = v.x;
      d[i + 1] = v.y;
      d[i + 2] = v.z;
      d[i + 3] = v.w;
    }
  }
  __syncwarp();  // rtot
  float t[8];
#pragma unroll
  for (int i = 0; i < 8; i += 4) {
    const float4 r4 = *(const float4*)(rtot + 8 * (lane >> 3) + i);
    t[i] = r4.x;
    t[i + 1] = r4.y;
    t[i + 2] = r4.z;
    t[i + 3] = r4.w;
  }
#pragma unroll
  for (int i = 0; i < 8; i++) {
    t[i] = __fmul_rn(__fmul_rn(d[i], d[i]), t[i]);
    accm[i] = fmaf(wm, t[i], accm[i]);
    accg[i] = fmaf(wg, t[i], accg[i]);
  }
  if constexpr (kRaw) {
#pragma unroll
    for (int i = 0; i < 8; i++) t[i] += __shfl_xor_sync(FULL, t[i], 16);
#pragma unroll
    for (int i = 0; i < 8; i++) t[i] += __shfl_xor_sync(FULL, t[i], 8);
    const float chi = 0.5f * (((t[0] + t[4]) + (t[2] + t[6])) + ((t[1] + t[5]) + (t[3] + t[7])));
    if (lane < 8) raw[lane * raw_stride] = chi;
  }
}

// What bounds it: the shared-memory pipe and instruction issue, about evenly
// (the bytes are nothing: 4 in + 64 out per pixel).
template <bool kRaw>
__global__ void __launch_bounds__(CT_WARPS * 32, 3) k_cues(const PatchDev* __restrict__ patches,
                                                        const int4* __restrict__ work,
                                                        const uint32_t* __restrict__ lab4,
                                                        const int* __restrict__ nbins,
                                                        float* __restrict__ mpbo, float* __restrict__ go,
                                                        float* __restrict__ raw, uint8_t* __restrict__ counts) {
  extern __shared__ __align__(16) uint8_t smem[];
  uint32_t* tile = (uint32_t*)smem;
  int16_t* offs = (int16_t*)(smem + CT_OFFS);  // [kAnnRows][32]
  const int4 w = work[blockIdx.x];
  const PatchDev P = patches[w.x];
  const uint32_t* lb = lab4 + P.pix;
  for (int i = threadIdx.x; i < CT_PH * CT_PW; i += blockDim.x) {
    const int yy = reflect_c(w.y - kMaxRadius + i / CT_PW, P.H);
    const int xx = reflect_c(w.z - kMaxRadius + i % CT_PW, P.W);
    tile[i] = lb[(long long)yy * P.W + xx];
  }
  // disc offsets, entry i of every lane's list side by side: annulus a of
  // lane l starts at row c_ann_row[a]
  for (int i = threadIdx.x; i < c_ann_row[kNannulus] * 32; i += blockDim.x) {
    const int r = i >> 5, l = i & 31;
    int a = 0;
    while (r >= c_ann_row[a + 1]) a++;
    const int k = r - c_ann_row[a];
    if (k < c_ann_count[a][l]) {
      const int e = c_ann_start[a][l] + k;
      offs[i] = (int16_t)(c_ann_dy[e] * CT_PW + c_ann_dx[e]);
    }
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint8_t* hist = smem + CT_HIST + warp * HWARP;
  float* dsm = (float*)(smem + CT_ROWS) + warp * DWARP;
  for (int i = lane; i < DWARP; i += 32) dsm[i] = 0.f;  // the rows' zero margins
  __syncthreads();
  const int nbL = nbins[4 * w.x + 0] + 1, nbA = nbins[4 * w.x + 1] + 1, nbB = nbins[4 * w.x + 2] + 1,
            nbT = nbins[4 * w.x + 3] + 1;
  const float mL = bin_mass<17>(c_kbg, lane, nbL);
  const float mA = bin_mass<9>(c_kcg, lane, nbA);
  const float mB = bin_mass<9>(c_kcg, lane, nbB);
  const int y = w.y + warp;
  if (y >= P.H) return;
  uint8_t* r0 = hist + lane;
  uint8_t* r1 = r0 + HCUE;
  uint8_t* r2 = r1 + HCUE;
  uint8_t* r3 = r2 + HCUE;
  for (int px = 0; px < CT_W; px++) {
    const int x = w.z + px;
    if (x >= P.W) break;
    const long long p = (long long)y * P.W + x;
#pragma unroll
    for (int c = 0; c < 4; c++)
      if (c == 3 || lane < kLabBins) {
        uint4* bin = (uint4*)(hist + c * HCUE + lane * HPITCH);
        bin[0] = make_uint4(0u, 0u, 0u, 0u);
        bin[1] = make_uint4(0u, 0u, 0u, 0u);
      }
    __syncwarp();
    const uint32_t* ctr = tile + (warp + kMaxRadius) * CT_PW + (px + kMaxRadius);
    float accm[8], accg[8];
#pragma unroll
    for (int o = 0; o < 8; o++) accm[o] = accg[o] = 0.f;
    const long long rs = P.N;
#pragma unroll 1
    for (int a = 0; a < kNannulus; a++) {
      const int cnt = c_ann_count[a][lane];
      const int16_t* of = offs + c_ann_row[a] * 32 + lane;
      if (a < 3) {
        for (int i = 0; i < cnt; i++) {
          const uint32_t v = ctr[of[32 * i]];
          r0[(v & 255) * HPITCH]++;
          r1[((v >> 8) & 255) * HPITCH]++;
          r2[((v >> 16) & 255) * HPITCH]++;
          r3[(v >> 24) * HPITCH]++;
        }
      } else {
        for (int i = 0; i < cnt; i++) {
          const uint32_t v = ctr[of[32 * i]];
          r1[((v >> 8) & 255) * HPITCH]++;
          r2[((v >> 16) & 255) * HPITCH]++;
          r3[(v >> 24) * HPITCH]++;
        }
      }
      __syncwarp();
      if (kRaw && counts) {
        // debug: this lane's counter rows (half = lane / 16, slice = lane % 16)
        uint8_t* cp = counts + (((P.pix + p) * kNannulus + a) * 4) * 32 * 32;
#pragma unroll
        for (int c = 0; c < 4; c++)
          for (int bb = 0; bb < 32; bb++)
            cp[(c * 32 + lane) * 32 + bb] = (c == 3 || bb < kLabBins) ? hist[c * HCUE + bb * HPITCH + lane] : 0;
      }
      // cue index wi = cue*3 + scale (bg1 bg2 bg3 cga1 .. tg3)
      float* rawp = kRaw ? raw + P.pix * 96 + p : nullptr;
      if (a < 3)
        cue_combo<17, kRaw>(hist, lane, nbL, a, c_kbg, mL, c_wm[a], c_wg[a], accm, accg, rawp + (long long)a * 8 * rs,
                            rs, dsm);
      if (a > 0) {
        const int s = a - 1;  // scale of cga/cgb/tg
#pragma unroll 1
        for (int c = 1; c < 3; c++)
          cue_combo<9, kRaw>(hist + c * HCUE, lane, c == 1 ? nbA : nbB, a, c_kcg, c == 1 ? mA : mB, c_wm[3 * c + s],
                             c_wg[3 * c + s], accm, accg, rawp + (long long)(3 * c + s) * 8 * rs, rs, dsm);
        cue_combo<0, kRaw>(hist + 3 * HCUE, lane, nbT, a, nullptr, 0.f, c_wm[9 + s], c_wg[9 + s], accm, accg,
                           rawp + (long long)(9 + s) * 8 * rs, rs, dsm);
      }
      __syncwarp();
    }
    // sums over the bins: bits 4 and 3 of the bin are the lane's group, bits
    // 2..0 the register.  Lanes 0-15 keep the first weight set, 16-31 the
    // second; group bit 0 is added on both of its lanes.
    const bool hi = lane & 16;
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const float keep = hi ? accg[i] : accm[i], give = hi ? accm[i] : accg[i];
      v[i] = keep + __shfl_xor_sync(FULL, give, 16);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] += __shfl_xor_sync(FULL, v[i], 8);
    const float sum = ((v[0] + v[4]) + (v[2] + v[6])) + ((v[1] + v[5]) + (v[3] + v[7]));
    if (!(lane & 8)) (hi ? go : mpbo)[P.pix * 8 + (long long)(lane & 7) * P.N + p] = 0.5f * sum;
  }
}

// max label per patch and cue (the histogram length of hist_gradient_2D is
// max(label)+1, lib_image.cc:3665-3670)
__global__ void k_maxlabel(const PatchDev* __restrict__ patches, const uint32_t* __restrict__ lab4,
                           int* __restrict__ nbins) {
  const PatchDev P = patches[blockIdx.y];
  int m0 = 0, m1 = 0, m2 = 0, m3 = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < P.N; i += (long long)gridDim.x * blockDim.x) {
    const uint32_t v = lab4[P.pix + i];
    m0 = max(m0, (int)(v & 255));
    m1 = max(m1, (int)((v >> 8) & 255));
    m2 = max(m2, (int)((v >> 16) & 255));
    m3 = max(m3, (int)(v >> 24));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    m0 = max(m0, __shfl_xor_sync(FULL, m0, o));
    m1 = max(m1, __shfl_xor_sync(FULL, m1, o));
    m2 = max(m2, __shfl_xor_sync(FULL, m2, o));
    m3 = max(m3, __shfl_xor_sync(FULL, m3, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(&nbins[4 * blockIdx.y + 0], m0);
    atomicMax(&nbins[4 * blockIdx.y + 1], m1);
    atomicMax(&nbins[4 * blockIdx.y + 2], m2);
    atomicMax(&nbins[4 * blockIdx.y + 3], m3);
  }
}

// ---------------------------------------------------------------- NMS
__device__ __forceinline__ void argmax8(const float* __restrict__ mo, long long N, long long p,
                                        float& a, int& ind) {
  float mv = -FLT_MAX;
  int mi = 0;
#pragma unroll
  for (int o = 0; o < 8; o++) {
    const float d = mo[o * N + p];
    if (d > mv) {
      mv = d;
      mi = o;
    }
  }
  a = mv < 0.f ? 0.f : mv;
  ind = mi;
}

__global__ void __launch_bounds__(256) k_nms(const PatchDev* __restrict__ patches,
                                             const int4* __restrict__ work, const float* __restrict__ mpbo,
                                             float* __restrict__ mpb) {
  const int4 w = work[blockIdx.x];
  const PatchDev P = patches[w.x];
  const int y = w.y + threadIdx.x / 16, x = w.z + threadIdx.x % 16;
  if (y >= P.H || x >= P.W) return;
  const float* mo = mpbo + P.pix * 8;
  const long long N = P.N, p = (long long)y * P.W + x;
  float v;
  int i;
  argmax8(mo, N, p, v, i);
  // x of lib_image is the row, y the column
  float out = 0.f;
  bool ok = true;
  int nr[4], nc[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    nr[k] = y + c_nms_nb[i][k][0];
    nc[k] = x + c_nms_nb[i][k][1];
    ok = ok && nr[k] >= 0 && nr[k] < P.H && nc[k] >= 0 && nc[k] < P.W;
  }
  if (ok) {
    float va[4];
    int ia[4];
#pragma unroll
    for (int k = 0; k < 4; k++) argmax8(mo, N, (long long)nr[k] * P.W + nc[k], va[k], ia[k]);
    const float d = c_nms_d[i];
    const float v0 = (1.0f - d) * va[0] * c_nms_cos[i][ia[0]] + d * va[1] * c_nms_cos[i][ia[1]];
    const float v1 = (1.0f - d) * va[2] * c_nms_cos[i][ia[2]] + d * va[3] * c_nms_cos[i][ia[3]];
    if (v > v0 && v > v1) out = v;
  }
  // clip of multiscalePb.cpp:249-261 with the x1.2 of MATLAB's max(0,min(1,1.2 v)) (D7)
  out = (1.2f * out > 1.f) ? 1.f : 1.2f * out;
  if (out < 0.f) out = 0.f;
  mpb[P.pix + p] = out;
}

cudaError_t launch_maxlabel(const PatchDev* patches, int npatch, const uint32_t* lab4, int* nbins,
                            cudaStream_t s) {
  cudaMemsetAsync(nbins, 0, sizeof(int) * 4 * npatch, s);
  dim3 g(16, npatch);
  k_maxlabel<<<g, 256, 0, s>>>(patches, lab4, nbins);
  return cudaGetLastError();
}

cudaError_t launch_cues(const PatchDev* patches, const int4* work, int nwork, const uint32_t* lab4,
                        const int* nbins, float* mpbo, float* go, float* raw, uint8_t* counts, cudaStream_t s) {
  static PerDevice ready;
  const cudaError_t e = ready.once([] {
    const cudaError_t f = grant_smem(k_cues<false>, kCueSmem);
    return f != cudaSuccess ? f : grant_smem(k_cues<true>, kCueSmem);
  });
  if (e != cudaSuccess || nwork == 0) return e;
  if (raw)
    k_cues<true><<<nwork, CT_WARPS * 32, kCueSmem, s>>>(patches, work, lab4, nbins, mpbo, go, raw, counts);
  else
    k_cues<false><<<nwork, CT_WARPS * 32, kCueSmem, s>>>(patches, work, lab4, nbins, mpbo, go, raw, nullptr);
  return cudaGetLastError();
}

cudaError_t launch_nms(const PatchDev* patches, const int4* work, int nwork, const float* mpbo,
                       float* mpb, cudaStream_t s) {
  if (nwork == 0) return cudaSuccess;
  k_nms<<<nwork, 256, 0, s>>>(patches, work, mpbo, mpb);
  return cudaGetLastError();
}

}  // namespace gpb
