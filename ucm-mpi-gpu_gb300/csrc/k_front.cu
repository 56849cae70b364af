// k_front.cu -- colour conversion and Schmid textons (sm_103a).
//
// (1) convert: packed B<<16|G<<8|R (src/globalPb.cpp:264-276) -> 8-bit grey
//     (CV_BGR2GRAY, src/SPFeatures.cpp:27) and the 25-bin L, a, b labels of
//     mex_pb_parts_final_selected.cpp:97-134 (lib_image.cc:123-343).
// (2) texton: the 13 S filters (49x49, src/SPFeatures.cpp:117-183) correlated
//     with the reflect-padded grey image and the nearest of K codewords
//     (src/SPFeatures.cpp:277-360, argmin fixed).  The S filters are radial,
//     so the window folds into 325 symmetric groups (|dy|,|dx|) whose integer
//     pixel sums are exact; the 13 responses and the 32 distances run in FP32
//     with an error bound.  A pixel whose best and second-best distances are
//     closer than the bound goes to (3).
// (3) texton_repair: one CTA per flagged pixel recomputes the responses in
//     FP64 over radius rings in ascending order with unfused multiply/add --
//     the exact arithmetic of the FP64 restatement -- so labels are identical.
#include <math.h>
#include <stdint.h>

#include "f32x2.h"
#include "gpb_internal.h"
#include "kernels.h"

namespace gpb {

// Texton tile: 16 x 16 outputs and a halo of 24, rows of 80 bytes (a warp's 8
// rows x 4 words reach distinct banks), in four copies shifted by 0..3 bytes,
// so the 4 pixels at any displacement are one aligned word of one copy.
constexpr int TX_T = 16, TX_W = TX_T + 2 * 24, TX_PITCH = 80, TX_COPY = TX_W * TX_PITCH;
constexpr int kFilt = 16;    // filters per group in the weight table (13, padded)
constexpr int kChunk = 8;    // groups summed before they join the response
constexpr int kChunks = (kSchmidGroups + kChunk - 1) / kChunk;

constexpr int kGroupsPad = kChunks * kChunk;

__device__ __align__(16) float g_k32[kGroupsPad][kFilt];
__device__ float g_gammaf[256];
// the byte offsets, in the four copies, of a group's displacements: 8, or 4 in
// the first half and none in the second (bit of c_gmask[chunk] clear).  The
// centre counts 4 times with a quarter of its weight (exact); the groups past
// the last have zero weights.
__constant__ int4 c_goff[kGroupsPad][2];
__constant__ uint32_t c_gmask[kChunks];
__constant__ float c_codebook[kNschmid][kMaxCodewords];
__constant__ float c_errb[kNschmid];    // a-priori part of a response's error bound
__constant__ double c_gamma[256];
__constant__ int c_K;

void upload_front(const HostTables& t, cudaStream_t s) {
  float kt[kGroupsPad][kFilt] = {};
  int start[kSchmidGroups + 1];
  int8_t dy[2401], dx[2401];
  int n = 0;
  for (int g = 0; g < kSchmidGroups; g++) {
    start[g] = n;
    const int a = t.group_a[g], b = t.group_b[g];
    int cand[8][2] = {{a, b}, {a, -b}, {-a, b}, {-a, -b}, {b, a}, {b, -a}, {-b, a}, {-b, -a}};
    for (int i = 0; i < 8; i++) {
      bool dup = false;
      for (int j = start[g]; j < n; j++)
        if (dy[j] == cand[i][0] && dx[j] == cand[i][1]) dup = true;
      if (dup) continue;
      dy[n] = (int8_t)cand[i][0];
      dx[n] = (int8_t)cand[i][1];
      n++;
    }
    for (int f = 0; f < kNschmid; f++) kt[g][f] = t.k32_group[f][g] * (n - start[g] == 1 ? 0.25f : 1.f);
  }
  start[kSchmidGroups] = n;
  cudaMemcpyToSymbolAsync(g_k32, kt, sizeof(kt), 0, cudaMemcpyHostToDevice, s);
  int off[kGroupsPad][8] = {};
  uint32_t mask[kChunks] = {};
  for (int g = 0; g < kSchmidGroups; g++) {
    const int cnt = start[g + 1] - start[g];
    for (int i = 0; i < 8; i++) {
      const int j = start[g] + (i < cnt ? i : 0);
      const int o = dy[j] * TX_PITCH + dx[j], sh = o & 3;
      off[g][i] = o - sh + sh * TX_COPY;
    }
    if (cnt == 8) mask[g / kChunk] |= 1u << (g % kChunk);
  }
  cudaMemcpyToSymbolAsync(c_goff, off, sizeof(off), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_gmask, mask, sizeof(mask), 0, cudaMemcpyHostToDevice, s);
  // in-chunk rounding: each of a chunk's kChunk partial sums is at most the
  // chunk's sum of |weight| x (255 x pixels of the group)
  float errb[kNschmid];
  for (int f = 0; f < kNschmid; f++) {
    double l1 = 0;
    for (int g = 0; g < kSchmidGroups; g++) l1 += fabs((double)t.k32_group[f][g]) * (start[g + 1] - start[g]);
    errb[f] = (float)(kChunk * 255.0 * l1);
  }
  cudaMemcpyToSymbolAsync(c_errb, errb, sizeof(errb), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_gamma, t.gamma_lut, sizeof(t.gamma_lut), 0, cudaMemcpyHostToDevice, s);
  float gf[256];
  for (int i = 0; i < 256; i++) gf[i] = (float)t.gamma_lut[i];
  cudaMemcpyToSymbolAsync(g_gammaf, gf, sizeof(gf), 0, cudaMemcpyHostToDevice, s);
}

void upload_codebook(const float* cb, int K, cudaStream_t s) {
  float tmp[kNschmid][kMaxCodewords] = {};
  for (int f = 0; f < kNschmid; f++)
    for (int k = 0; k < K; k++) tmp[f][k] = cb[f * K + k];
  cudaMemcpyToSymbolAsync(c_codebook, tmp, sizeof(tmp), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_K, &K, sizeof(int), 0, cudaMemcpyHostToDevice, s);
}

__device__ __forceinline__ int reflect(int i, int n) {
  // BORDER_REFLECT (edge repeated); patches are >= 32 px so one fold suffices
  // for every padding used here, the loop is bounded by the two folds
  for (int it = 0; it < 4 && (i < 0 || i >= n); it++) i = (i < 0) ? -i - 1 : 2 * n - 1 - i;
  return i < 0 ? 0 : (i >= n ? n - 1 : i);
}

// ---------------------------------------------------------------- convert
// Lab chain with no fused multiply-add, in the order of the reference:
// gamma (table of pow(u/255, 2.5)), rgb_to_xyz, xyz_to_lab, lab_normalize,
// quantize_values (floor(v*25), 25 -> 24).
__device__ __forceinline__ int quant25(double v, int nbins) {
  if (v < 0) v = 0;
  else if (v > 1) v = 1;
  int q = (int)floor(__dmul_rn(v, (double)nbins));
  return q == nbins ? nbins - 1 : q;
}

// The bin of t = 25 v in FP32, or -1 where t is within m of a bin edge, so the
// FP64 chain has to decide (below 1 and above 24 the clamps make one bin of
// both sides)
__device__ __forceinline__ int bin_or_edge(float t, float m) {
  const float k = rintf(t);
  if (fabsf(t - k) < m && k >= 1.f && k <= 24.f) return -1;
  return min(max((int)floorf(t), 0), 24);
}
// The chain below in FP32; false where a value is too near an edge.  Errors:
// the tristimulus values are off by at most 4e-7, the cube roots by 3e-7, so
// t is off by at most 9e-6 (L), 4.5e-5 (a: 500 x 25 / 168 of two roots) and
// 1.8e-5 (b); the margins leave a factor of 3 and more.
__device__ __forceinline__ bool lab_bins_fast(int R, int G, int B, uint32_t& bins) {
  const float r = g_gammaf[R], g = g_gammaf[G], b = g_gammaf[B];
  const float x = (0.412453f * r + 0.357580f * g + 0.180423f * b) * (float)(1.0 / 0.950456);
  const float y = 0.212671f * r + 0.715160f * g + 0.072169f * b;
  const float z = (0.019334f * r + 0.119193f * g + 0.950227f * b) * (float)(1.0 / 1.088754);
  const float th = 0.008856f, c16 = (float)(16.0 / 116.0);
  if (fminf(fminf(fabsf(x - th), fabsf(y - th)), fabsf(z - th)) < 2e-6f) return false;  // either branch
  const float fx = x > th ? cbrtf(x) : fmaf(7.787f, x, c16);
  const float fy = y > th ? cbrtf(y) : fmaf(7.787f, y, c16);
  const float fz = z > th ? cbrtf(z) : fmaf(7.787f, z, c16);
  const float L = y > th ? 116.f * fy - 16.f : 903.3f * y;
  const int qL = bin_or_edge(L * 0.25f, 1e-4f);
  const int qa = bin_or_edge((500.f * (fx - fy) + 73.f) * (25.f / 168.f), 1.5e-4f);
  const int qb = bin_or_edge((200.f * (fy - fz) + 73.f) * (25.f / 168.f), 1e-4f);
  bins = (uint32_t)qL | ((uint32_t)qa << 8) | ((uint32_t)qb << 16);
  return qL >= 0 && qa >= 0 && qb >= 0;
}

// Lab bins (L | a << 8 | b << 16) of one BGR colour.  FP64 cube roots run at a
// small fraction of the FP32 rate: 1 Mpx took 803 us in FP64 alone, 42 us this
// way (about 0.1 % of the colours go to FP64).
__device__ __forceinline__ uint32_t lab_bins_of(int R, int G, int B) {
  uint32_t bins;
  if (lab_bins_fast(R, G, B, bins)) return bins;
  // D1 fixed: r = R, b = B
  const double r = c_gamma[R], g = c_gamma[G], b = c_gamma[B];
  const double X = __dadd_rn(__dadd_rn(__dmul_rn(0.412453, r), __dmul_rn(0.357580, g)), __dmul_rn(0.180423, b));
  const double Y = __dadd_rn(__dadd_rn(__dmul_rn(0.212671, r), __dmul_rn(0.715160, g)), __dmul_rn(0.072169, b));
  const double Z = __dadd_rn(__dadd_rn(__dmul_rn(0.019334, r), __dmul_rn(0.119193, g)), __dmul_rn(0.950227, b));
  const double x = __ddiv_rn(X, 0.950456), y = __ddiv_rn(Y, 1.000000), z = __ddiv_rn(Z, 1.088754);
  const double th = 0.008856, third = 1.0 / 3.0, c16 = 16.0 / 116.0;
  const double fx = (x > th) ? pow(x, third) : __dadd_rn(__dmul_rn(7.787, x), c16);
  const double fy = (y > th) ? pow(y, third) : __dadd_rn(__dmul_rn(7.787, y), c16);
  const double fz = (z > th) ? pow(z, third) : __dadd_rn(__dmul_rn(7.787, z), c16);
  const double L = (y > th) ? __dsub_rn(__dmul_rn(116.0, pow(y, third)), 16.0) : __dmul_rn(903.3, y);
  const double A = __dmul_rn(500.0, __dsub_rn(fx, fy));
  const double Bb = __dmul_rn(200.0, __dsub_rn(fy, fz));
  const int qL = quant25(__ddiv_rn(L, 100.0), 25);
  const int qa = quant25(__ddiv_rn(__dsub_rn(A, -73.0), 168.0), 25);
  const int qb = quant25(__ddiv_rn(__dsub_rn(Bb, -73.0), 168.0), 25);
  return (uint32_t)qL | ((uint32_t)qa << 8) | ((uint32_t)qb << 16);
}

__device__ __forceinline__ uint8_t grey_of(int R, int G, int B) {
  return (uint8_t)((R * 4899 + G * 9617 + B * 1868 + (1 << 13)) >> 14);
}

__global__ void __launch_bounds__(256) k_convert(const uint32_t* __restrict__ packed, long long n,
                                                 uint8_t* __restrict__ grey,
                                                 uint32_t* __restrict__ lab4) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t px = packed[i];
  const int B = (px >> 16) & 255, G = (px >> 8) & 255, R = px & 255;
  grey[i] = grey_of(R, G, B);
  lab4[i] = lab_bins_of(R, G, B);
}

// The Lab bins of all 2^24 colours, indexed by the packed value B<<16|G<<8|R:
// the pipeline's convert step then gathers from this table (FP64 cube roots
// run at a small fraction of the FP32 rate on this part).
__global__ void __launch_bounds__(256) k_lab_table(uint32_t* __restrict__ table) {
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < (1u << 24); c += gridDim.x * blockDim.x)
    table[c] = lab_bins_of(c & 255, (c >> 8) & 255, c >> 16);
}

__global__ void __launch_bounds__(256) k_convert_lut(const uint32_t* __restrict__ packed, long long n,
                                                     const uint32_t* __restrict__ table,
                                                     uint8_t* __restrict__ grey, uint32_t* __restrict__ lab4) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t px = packed[i];
  grey[i] = grey_of(px & 255, (px >> 8) & 255, (px >> 16) & 255);
  lab4[i] = __ldg(table + (px & 0xffffffu));
}

// ----------------------------------------------------------------- texton
// 64 threads cover a 16 x 16 tile, a thread 4 horizontally adjacent pixels
// (pairs of bytes in 16-bit halves: a group's sum is at most 8 x 255), and
// SPLIT such sets of threads share the groups, for launches of few tiles.
// The 13 responses are packed FP32 FMA chains over chunks of kChunk groups,
// each chunk's sum then added to the response, so the error bound
//   |error of R_f| <= u (sum over adds of |R_f| + c_errb[f])
// (u = 2^-24) costs one add per chunk instead of one per group; the thread's
// four pixels share it (the largest |R_f| counts).  Split responses are added
// in order, each add entering the bound too.  The split
// moves a response within its bound; labels that the bound leaves open are
// decided in FP64 (k_texton_repair), so every split gives the same labels and
// the autotuner picks among them.
// Bound by instruction issue: per group and 4 pixels 8 words (a load and four
// integer operations each) and 26 packed FMAs.  Measured: 534 us for 1024^2
// (741 with scalar sums, FMAs and a bound per group), 34 us for 96 x 131 with
// SPLIT = 4 (128 with one set of threads per tile).  Merging the groups of
// equal length (273 rings) saved FMAs but its branches cost more: 733 us.
template <int SPLIT>
__global__ void __launch_bounds__(64 * SPLIT) k_texton(const PatchDev* __restrict__ patches,
                                                       const int4* __restrict__ work,
                                                       const uint8_t* __restrict__ grey,
                                                       uint32_t* __restrict__ lab4, int* __restrict__ repair_list,
                                                       int* __restrict__ repair_count, int repair_cap) {
  constexpr int NV = kNschmid * 5;  // a thread's responses and bounds
  __shared__ __align__(16) unsigned char sm[4 * TX_COPY + sizeof(float) * kGroupsPad * kFilt];
  static_assert(NV * 64 * sizeof(float) <= sizeof(sm), "exchange of split responses");
  uint32_t* copies = (uint32_t*)sm;
  const float4* kt = (const float4*)(sm + 4 * TX_COPY);
  const int4 w = work[blockIdx.x];  // (patch, ty0, tx0, -)
  const PatchDev P = patches[w.x];
  const uint8_t* g = grey + P.pix;
  for (int i = threadIdx.x; i < TX_W * TX_PITCH; i += blockDim.x) {
    const int r = i / TX_PITCH, q = i % TX_PITCH;
    uint8_t v = 0;
    if (q < TX_W) v = g[(long long)reflect(w.y - 24 + r, P.H) * P.W + reflect(w.z - 24 + q, P.W)];
    sm[i] = v;
  }
  for (int i = threadIdx.x; i < kGroupsPad * kFilt / 4; i += blockDim.x)
    ((float4*)(sm + 4 * TX_COPY))[i] = ((const float4*)g_k32)[i];
  __syncthreads();
  constexpr int NW = TX_COPY / 4;
  for (int i = threadIdx.x; i < NW; i += blockDim.x) {
    const uint32_t w0 = copies[i], w1 = i + 1 < NW ? copies[i + 1] : 0u;
#pragma unroll
    for (int sh = 1; sh < 4; sh++) copies[sh * NW + i] = __funnelshift_r(w0, w1, 8 * sh);
  }
  __syncthreads();
  const int set = threadIdx.x >> 6, t = threadIdx.x & 63, ty = t >> 2, tx = 4 * (t & 3);
  F2 R[kNschmid][2];
  float E[kNschmid];
#pragma unroll
  for (int f = 0; f < kNschmid; f++) {
    R[f][0] = R[f][1] = f2(0.f, 0.f);
    E[f] = 0.f;
  }
  const unsigned char* c = sm + (ty + 24) * TX_PITCH + tx + 24;
#pragma unroll 1
  for (int m = kChunks * set / SPLIT; m < kChunks * (set + 1) / SPLIT; m++) {
    F2 r[kNschmid][2];
#pragma unroll
    for (int f = 0; f < kNschmid; f++) r[f][0] = r[f][1] = f2(0.f, 0.f);
    const uint32_t mask = c_gmask[m];
#pragma unroll 1
    for (int u0 = 0; u0 < kChunk; u0 += 4) {  // the words of 4 groups in flight, then their FMAs
      const int g0 = m * kChunk + u0;
      uint32_t even[4], odd[4];  // 16-bit sums of pixels 0, 2 and 1, 3
#pragma unroll
      for (int u = 0; u < 4; u++) {
        even[u] = odd[u] = 0;
        auto add4 = [&](const int4& o) {
          const uint32_t v0 = *(const uint32_t*)(c + o.x), v1 = *(const uint32_t*)(c + o.y);
          const uint32_t v2 = *(const uint32_t*)(c + o.z), v3 = *(const uint32_t*)(c + o.w);
          even[u] += (v0 & 0x00ff00ffu) + (v1 & 0x00ff00ffu);
          even[u] += (v2 & 0x00ff00ffu) + (v3 & 0x00ff00ffu);
          odd[u] += __byte_perm(v0, 0, 0x4341) + __byte_perm(v1, 0, 0x4341);
          odd[u] += __byte_perm(v2, 0, 0x4341) + __byte_perm(v3, 0, 0x4341);
        };
        add4(c_goff[g0 + u][0]);
        if (mask >> (u0 + u) & 1u) add4(c_goff[g0 + u][1]);
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const F2 s0 = f2((float)(even[u] & 0xffffu), (float)(odd[u] & 0xffffu));
        const F2 s1 = f2((float)(even[u] >> 16), (float)(odd[u] >> 16));
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const float4 k4 = kt[(g0 + u) * (kFilt / 4) + q];
          const float kf[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
          for (int v = 0; v < 4; v++) {
            const int f = 4 * q + v;
            if (f >= kNschmid) break;
            const F2 kk = f2(kf[v], kf[v]);
            r[f][0] = f2_fma(kk, s0, r[f][0]);
            r[f][1] = f2_fma(kk, s1, r[f][1]);
          }
        }
      }
    }
#pragma unroll
    for (int f = 0; f < kNschmid; f++) {
      R[f][0] = f2_add(R[f][0], r[f][0]);
      R[f][1] = f2_add(R[f][1], r[f][1]);
      const float2 v = f2_split(R[f][0]), w2 = f2_split(R[f][1]);
      E[f] += fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(w2.x), fabsf(w2.y)));
    }
  }
  float Rv[kNschmid][4];
#pragma unroll
  for (int f = 0; f < kNschmid; f++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const float2 v = f2_split(R[f][h]);
      Rv[f][2 * h] = v.x;
      Rv[f][2 * h + 1] = v.y;
    }
  constexpr int NP = 4 / SPLIT;  // pixels that each set decides
  float* ex = (float*)sm;        // [NV][64]
  if constexpr (SPLIT > 1) {
    auto give = [&]() {
#pragma unroll
      for (int f = 0; f < kNschmid; f++) {
#pragma unroll
        for (int k = 0; k < 4; k++) ex[(f * 5 + k) * 64 + t] = Rv[f][k];
        ex[(f * 5 + 4) * 64 + t] = E[f];
      }
    };
    for (int from = 1; from < SPLIT; from++) {
      __syncthreads();
      if (set == from) give();
      __syncthreads();
      if (set == 0) {
#pragma unroll
        for (int f = 0; f < kNschmid; f++) {
          float most = 0.f;
#pragma unroll
          for (int k = 0; k < 4; k++) {
            Rv[f][k] += ex[(f * 5 + k) * 64 + t];
            most = fmaxf(most, fabsf(Rv[f][k]));
          }
          E[f] += ex[(f * 5 + 4) * 64 + t] + most;
        }
      }
    }
    __syncthreads();
    if (set == 0) give();
    __syncthreads();
  }
  const int K = c_K;
#pragma unroll
  for (int kp = 0; kp < NP; kp++) {
    const int k = NP * set + kp;
    const int y = w.y + ty, x = w.z + tx + k;
    if (y >= P.H || x >= P.W) continue;
    float Rp[kNschmid], Ep[kNschmid];
#pragma unroll
    for (int f = 0; f < kNschmid; f++) {
      Rp[f] = SPLIT > 1 ? ex[(f * 5 + k) * 64 + t] : Rv[f][kp];
      Ep[f] = SPLIT > 1 ? ex[(f * 5 + 4) * 64 + t] : E[f];
      Ep[f] = (Ep[f] + c_errb[f]) * 6.0e-8f * 1.01f + 1e-6f;
    }
    float d1 = 3.4e38f, d2 = 3.4e38f;
    int k1 = 0, k2 = 0;
    for (int q = 0; q < K; q++) {
      float d = 0.f;
#pragma unroll
      for (int f = 0; f < kNschmid; f++) {
        const float u = Rp[f] - c_codebook[f][q];
        d = fmaf(u, u, d);
      }
      if (d < d1) {
        d2 = d1;
        k2 = k1;
        d1 = d;
        k1 = q;
      } else if (d < d2) {
        d2 = d;
        k2 = q;
      }
    }
    // error bound of d(k1) and d(k2): responses off by at most Ep each, plus
    // the FP32 rounding of the distance sums themselves
    float margin = 0.f;
#pragma unroll
    for (int f = 0; f < kNschmid; f++) {
      const float eb = Ep[f];
      margin += 2.f * eb * (fabsf(Rp[f] - c_codebook[f][k1]) + fabsf(Rp[f] - c_codebook[f][k2]) + eb);
    }
    margin = 2.f * margin + 4e-6f * (d1 + d2) + 1e-6f;
    const long long pix = P.pix + (long long)y * P.W + x;
    uint32_t v = lab4[pix] & 0x00ffffffu;
    lab4[pix] = v | ((uint32_t)k1 << 24);
    if (K > 1 && d2 - d1 <= margin) {
      const int slot = atomicAdd(repair_count, 1);
      if (slot < repair_cap) {
        repair_list[2 * slot] = w.x;
        repair_list[2 * slot + 1] = y * P.W + x;
      }
    }
  }
}

constexpr int kRingChunk = 69;  // odd: the 13 rows reach distinct banks
// FP64 repair, a CTA per flagged pixel: ring sums in integers, the products
// K32[f][r] * S[r] in parallel, then their sums in ascending ring order and
// the squared distances, all without contraction.  Bound by latency (a few
// pixels in a thousand): 24 us at 96 x 131 and 45 us at 1024^2, from 54 and 86
// us with a warp per pixel and one load at a time.  The first warp sums a chunk
// of rings while the others form the next chunk's products: with all products
// of a pixel in shared memory (30 KB) 7 CTAs fit an SM, and 1024^2 pixels that
// are all flagged (two equal codewords) take 67 ms; 39 ms in chunks, 59 ms with
// a warp per pixel.
__global__ void __launch_bounds__(128) k_texton_repair(const PatchDev* __restrict__ patches,
                                                       const uint8_t* __restrict__ grey,
                                                       uint32_t* __restrict__ lab4,
                                                       const int* __restrict__ repair_list,
                                                       const int* __restrict__ repair_count,
                                                       int repair_cap, const double* __restrict__ k32_ring,
                                                       const int* __restrict__ ring_of, int n_rings) {
  __shared__ double prod[2][kNschmid * kRingChunk];
  extern __shared__ int S[];  // [n_rings]
  __shared__ double Rsh[kNschmid];
  const int nch = (n_rings + kRingChunk - 1) / kRingChunk;
  const int tid = threadIdx.x, lane = tid & 31;
  const int total = min(*repair_count, repair_cap);
  for (int item = blockIdx.x; item < total; item += gridDim.x) {
    const PatchDev P = patches[repair_list[2 * item]];
    const int p = repair_list[2 * item + 1];
    const int y = p / P.W, x = p % P.W;
    for (int r = tid; r < n_rings; r += 128) S[r] = 0;
    __syncthreads();
    const uint8_t* g = grey + P.pix;
#pragma unroll 10
    for (int o = tid; o < 2401; o += 128) {
      const int dy = o / 49 - 24, dx = o % 49 - 24;
      const int v = g[(long long)reflect(y + dy, P.H) * P.W + reflect(x + dx, P.W)];
      atomicAdd(&S[ring_of[o]], v);
    }
    __syncthreads();
    // products of a chunk of rings, [filter][ring of the chunk]
    auto products = [&](int c, int t0, int nt) {
      const int r0 = c * kRingChunk, nr = min(kRingChunk, n_rings - r0);
#pragma unroll 8
      for (int e = t0; e < kNschmid * kRingChunk; e += nt) {
        const int f = e / kRingChunk, r = e % kRingChunk;
        if (r < nr) prod[c & 1][e] = __dmul_rn(k32_ring[f * n_rings + r0 + r], (double)S[r0 + r]);
      }
    };
    products(0, tid, 128);
    __syncthreads();
    double acc = 0;
    for (int c = 0; c < nch; c++) {
      if (tid >= 32) {
        if (c + 1 < nch) products(c + 1, tid - 32, 96);
      } else if (lane < kNschmid) {
        const int nr = min(kRingChunk, n_rings - c * kRingChunk);
#pragma unroll 8
        for (int r = 0; r < nr; r++) acc = __dadd_rn(acc, prod[c & 1][lane * kRingChunk + r]);
      }
      __syncthreads();
    }
    if (tid < 32) {
      if (lane < kNschmid) Rsh[lane] = acc;
      __syncwarp();
      const int K = c_K;
      double d = 1e300;
      if (lane < K) {
        d = 0;
        for (int f = 0; f < kNschmid; f++) {
          const double u = __dsub_rn(Rsh[f], (double)c_codebook[f][lane]);
          d = __dadd_rn(d, __dmul_rn(u, u));
        }
      }
      // argmin, first index on ties
      int best = lane;
      for (int off = 16; off > 0; off >>= 1) {
        const double od = __shfl_xor_sync(0xffffffffu, d, off);
        const int ob = __shfl_xor_sync(0xffffffffu, best, off);
        if (od < d || (od == d && ob < best)) {
          d = od;
          best = ob;
        }
      }
      if (lane == 0) {
        const long long pix = P.pix + p;
        lab4[pix] = (lab4[pix] & 0x00ffffffu) | ((uint32_t)best << 24);
      }
    }
    __syncthreads();
  }
}

cudaError_t launch_convert(const uint32_t* packed, long long n, uint8_t* grey, uint32_t* lab4,
                           cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  k_convert<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(packed, n, grey, lab4);
  return cudaGetLastError();
}
cudaError_t launch_lab_table(uint32_t* table, cudaStream_t s) {
  k_lab_table<<<4096, 256, 0, s>>>(table);
  return cudaGetLastError();
}
cudaError_t launch_convert_lut(const uint32_t* packed, long long n, const uint32_t* table, uint8_t* grey,
                               uint32_t* lab4, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  k_convert_lut<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(packed, n, table, grey, lab4);
  return cudaGetLastError();
}

cudaError_t launch_texton(const PatchDev* patches, const int4* work, int nwork, const uint8_t* grey,
                          uint32_t* lab4, int* repair_list, int* repair_count, int repair_cap,
                          cudaStream_t s, int variant) {
  if (nwork == 0) return cudaSuccess;
  if (variant == 0)
    k_texton<1><<<nwork, 64, 0, s>>>(patches, work, grey, lab4, repair_list, repair_count, repair_cap);
  else if (variant == 2)
    k_texton<4><<<nwork, 256, 0, s>>>(patches, work, grey, lab4, repair_list, repair_count, repair_cap);
  else
    k_texton<2><<<nwork, 128, 0, s>>>(patches, work, grey, lab4, repair_list, repair_count, repair_cap);
  return cudaGetLastError();
}

cudaError_t launch_texton_repair(const PatchDev* patches, const uint8_t* grey, uint32_t* lab4,
                                 const int* repair_list, const int* repair_count, int repair_cap,
                                 const double* k32_ring, const int* ring_of, int n_rings,
                                 cudaStream_t s) {
  k_texton_repair<<<1216, 128, n_rings * sizeof(int), s>>>(patches, grey, lab4, repair_list, repair_count, repair_cap,
                                                           k32_ring, ring_of, n_rings);
  return cudaGetLastError();
}

}  // namespace gpb
