// k_eig.cu -- batched Krylov-Schur (thick-restart Lanczos) kernels for the
// smallest eigenpairs of A = I - D^-1/2 W D^-1/2 (sm_103a).
//
// Reference: the Lanczos eigensolver of
// damascene/src/noReorthog/lanczos.cu:192-752 and the stencil SpMV of
// damascene/src/stencilMatrixMultiply/stencilMVM.cu:129-182; the CPU path's
// Spectra SymGEigsSolver (src/spectralPb.cpp:221-245) defines the problem.
//
// One Lanczos step for every active patch of the batch is three launches
//   ks_spmv   w = A v_j (FP32 symmetric stencil SpMV, the lower triangle read
//             as the upper array shifted by the offset), v_j = w_prev / beta
//             written on the fly, h = V^T w
//   ks_orth   w -= V h, h2 = V^T w          (classical Gram-Schmidt, pass 1)
//   ks_orth   w -= V h2, beta^2 = |w|^2     (pass 2)
// or, where the tiles of the batch leave SMs idle, five: ks_mult and
// ks_project form the first two w with a pixel or two per thread, and ks_dots
// takes the dots with the basis vectors dealt over several CTAs per tile.
// Dot products are FMA chains over a thread's pixels, summed across the
// warp and the CTA in float-float (a compensated FP32 pair; FP64 runs at
// 1/64 of the FP32 rate on this part); the first CGS pass's projection V h,
// whose subtraction cancels most of w on a converging step, is formed
// float-float with exact products.  The per-CTA partials are reduced in FP64
// by the last CTA of each patch to finish (threadfence + atomic counter), so
// no separate reduction launches.
// The projected matrix T lives in device memory; at the end of a restart
// cycle the host solves it (eig_host.cpp) and ks_restart assembles the kept
// Ritz vectors.
#include <stdint.h>

#include <algorithm>

#include "gpb_internal.h"
#include "kernels.h"
#include "f32x2.h"
#include "k_eig.h"

namespace gpb {

__constant__ int c_up_dy[kUpper], c_up_dx[kUpper];

void upload_eig(const HostTables& t, cudaStream_t s) {
  int dy[kUpper], dx[kUpper];
  for (int j = 0; j < kUpper; j++) {
    dy[j] = t.sdy[kStencilN / 2 + 1 + j];
    dx[j] = t.sdx[kStencilN / 2 + 1 + j];
  }
  cudaMemcpyToSymbolAsync(c_up_dy, dy, sizeof(dy), 0, cudaMemcpyHostToDevice, s);
  cudaMemcpyToSymbolAsync(c_up_dx, dx, sizeof(dx), 0, cudaMemcpyHostToDevice, s);
}

constexpr unsigned FULLM = 0xffffffffu;

__device__ __forceinline__ void ff_add_prod(float& hi, float& lo, float a, float b) {
  // __fmul_rn / __fadd_rn: never contracted into an FMA, which would break
  // the error-free transformations
  const float p = __fmul_rn(a, b);
  const float pe = fmaf(a, b, -p);
  const float s = __fadd_rn(hi, p);
  const float z = s - hi;
  const float e = (hi - (s - z)) + (p - z);
  hi = s;
  lo += e + pe;
}
// the same for two pixels at once
__device__ __forceinline__ void ff_add_prod2(F2& hi, F2& lo, F2 a, F2 b) {
  const F2 p = f2_mul(a, b);
  const F2 pe = f2_fma(a, b, f2_neg(p));
  const F2 s = f2_add(hi, p);
  const F2 z = f2_sub(s, hi);
  const F2 e = f2_add(f2_sub(hi, f2_sub(s, z)), f2_sub(p, z));
  hi = s;
  lo = f2_add(lo, f2_add(e, pe));
}
__device__ __forceinline__ void ff_add(float& hi, float& lo, float bhi, float blo) {
  const float s = hi + bhi;
  const float z = s - hi;
  const float e = (hi - (s - z)) + (bhi - z);
  hi = s;
  lo += e + blo;
}
// float-float sum over the warp, in FP32 (every lane gets it); the FP64
// pipe, about 1/64 of the FP32 rate here, is left to one conversion per CTA
__device__ __forceinline__ float2 ff_warp_reduce(float hi, float lo) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float h2 = __shfl_xor_sync(FULLM, hi, o), l2 = __shfl_xor_sync(FULLM, lo, o);
    ff_add(hi, lo, h2, l2);
  }
  return make_float2(hi, lo);
}

// Last CTA of a patch: returns true in every thread of that CTA.
__device__ __forceinline__ bool last_cta(int* counter, int ntiles) {
  __shared__ int is_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    const int prev = atomicAdd(counter, 1);
    is_last = (prev == ntiles - 1);
    if (is_last) *counter = 0;
  }
  __syncthreads();
  if (is_last) __threadfence();
  return is_last;
}

// basis vectors loaded together
constexpr int kGrp = 8;
// per-warp partial sums (sred[warp][i], written by lane 0) -> one partial per
// tile in part[tile][i], for the values i of the groups g, g + ng, ..
constexpr int kRed = kMaxKrylov + 1;
__device__ __forceinline__ void cta_partials(const float2* sred, int nvals, double* part_row, int g = 0, int ng = 1) {
  __syncthreads();
  for (int i = threadIdx.x; i < nvals; i += blockDim.x) {
    if (i / kGrp % ng != g) continue;
    float hi = 0.f, lo = 0.f;
#pragma unroll
    for (int w = 0; w < kEigWarps; w++) ff_add(hi, lo, sred[w * kRed + i].x, sred[w * kRed + i].y);
    part_row[i] = (double)hi + (double)lo;
  }
}
// The sums of values 0 .. n-1 over the CTAs of a patch, by the patch's last
// CTA: warp w takes the values w, w + 8, ...; each is a lane-strided FP64 sum
// and a tree over the warp.  put(i, sum, was) on one lane per value; was =
// before(i), loaded ahead.  This is the serial tail of every Lanczos launch
// (one CTA works, the other SMs wait for the next launch), so all loads of a
// warp's values are in flight together: one value at a time, each with its
// own loads, shuffles and read-modify-write of T, took 10 of the 26 us of a
// launch on one 321 x 481 image.
template <class B, class F>
__device__ __forceinline__ void patch_sums(const double* part, int tb, int tc, int mp1, int n, int warp, int lane,
                                           B&& before, F&& put) {
  constexpr int NI = (kMaxKrylov + 1 + kEigWarps - 1) / kEigWarps;
  double s[NI], was[NI];
#pragma unroll
  for (int u = 0; u < NI; u++) {
    const int i = warp + u * kEigWarps;
    s[u] = 0;
    was[u] = i < n ? before(i) : 0.0;
  }
  for (int b = tb + lane; b < tb + tc; b += 32) {
    double v[NI];
#pragma unroll
    for (int u = 0; u < NI; u++) {
      const int i = warp + u * kEigWarps;
      v[u] = i < n ? part[(long long)b * mp1 + i] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < NI; u++)
      if (warp + u * kEigWarps < n) s[u] += v[u];
  }
#pragma unroll
  for (int u = 0; u < NI; u++) {
    if (warp + u * kEigWarps >= n) break;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s[u] += __shfl_xor_sync(FULLM, s[u], o);
  }
  if (lane == 0) {
#pragma unroll
    for (int u = 0; u < NI; u++)
      if (warp + u * kEigWarps < n) put(warp + u * kEigWarps, s[u], was[u]);
  }
}

// Loads are issued in batches -- the stencil by offset for all eight pixels
// of a thread, the basis by groups of kGrp vectors -- so each thread keeps
// tens of independent loads in flight; every per-pixel sum still runs in the
// same order (offsets ascending, basis vectors ascending, pixels ascending).
// In the passes over the basis a load's address is a CTA-uniform base (array +
// vector + patch) plus the pixel's 32-bit byte offset in its patch (at most
// 2^28).  The stencil keeps 64-bit sums: with four uniform bases per offset it
// took 39 us instead of 26.
__device__ __forceinline__ float ldu(const float* base, uint32_t off) {
  return *(const float*)((const char*)base + off);
}
__device__ __forceinline__ void stu(float* base, uint32_t off, float v) { *(float*)((char*)base + off) = v; }
// the same on every lane; tells the compiler so
__device__ __forceinline__ long long uniform(long long v) {
  const uint32_t lo = __shfl_sync(FULLM, (uint32_t)v, 0), hi = __shfl_sync(FULLM, (uint32_t)(v >> 32), 0);
  return (long long)(((uint64_t)hi << 32) | lo);
}

// Sums kGrp = 8 float-float values over the warp at once.  Each of the first
// three xor rounds halves the values a lane carries (it keeps the half its
// lane bit selects and sends the other), the last two are plain: 18
// exchanges of a (hi, lo) pair and 9 float-float additions for the 8 values
// instead of 80 and 40.  Lane l ends with the total of value l >> 2.
__device__ __forceinline__ float2 ff_warp_reduce8(float (&hi)[kGrp], float (&lo)[kGrp], int lane) {
#pragma unroll
  for (int half = 4, o = 16; half >= 1; half >>= 1, o >>= 1) {
    const bool b = lane & o;
#pragma unroll
    for (int i = 0; i < half; i++) {
      const float kh = b ? hi[i + half] : hi[i], kl = b ? lo[i + half] : lo[i];
      const float gh = b ? hi[i] : hi[i + half], gl = b ? lo[i] : lo[i + half];
      hi[i] = kh;
      lo[i] = kl;
      ff_add(hi[i], lo[i], __shfl_xor_sync(FULLM, gh, o), __shfl_xor_sync(FULLM, gl, o));
    }
  }
#pragma unroll
  for (int o = 2; o >= 1; o >>= 1) ff_add(hi[0], lo[0], __shfl_xor_sync(FULLM, hi[0], o), __shfl_xor_sync(FULLM, lo[0], o));
  return make_float2(hi[0], lo[0]);
}

// h_i = v_i . w for i = 0..j, of the groups g, g + ng, .. of 8, over this
// thread's pixels (w is 0 at a pixel past the tile), reduced per warp into sred[warp][i]; v_j comes from
// registers (xj) when given.  A plain FMA chain over the thread's eight
// pixels, then float-float across threads: the error of a dot is a few
// units of rounding times |w| (Cauchy-Schwarz over the thread partials),
// which after the second pass leaves the basis orthogonal to ~1e-7 --
// two orders below what the Ritz residuals need.
__device__ __forceinline__ void basis_dots(const EigArgs& a, int j, long long base, const uint32_t (&qv)[kEigPix],
                                           const float (&wv)[kEigPix], const float* xj, float2* sred, int warp,
                                           int lane, int g = 0, int ng = 1) {
  for (int i0 = g * kGrp; i0 <= j; i0 += ng * kGrp) {
    float vv[kGrp][kEigPix];
#pragma unroll
    for (int u = 0; u < kGrp; u++) {
      const int i = i0 + u;
      const float* Vi = a.V + (long long)i * a.lvec + base;
#pragma unroll
      for (int r = 0; r < kEigPix; r++) vv[u][r] = (i < j || (i == j && !xj)) ? ldu(Vi, qv[r]) : (i == j ? xj[r] : 0.f);
    }
    float hi[kGrp], lo[kGrp];
#pragma unroll
    for (int u = 0; u < kGrp; u++) {
      hi[u] = lo[u] = 0.f;
#pragma unroll
      for (int r = 0; r < kEigPix; r++) hi[u] = fmaf(vv[u][r], wv[r], hi[u]);
    }
    const float2 sum = ff_warp_reduce8(hi, lo, lane);
    const int i = i0 + (lane >> 2);
    if ((lane & 3) == 0 && i <= j) sred[warp * kRed + i] = sum;
  }
}

// A patch's last CTA: its dots, into hbuf and T.  PASS 1 puts h; PASS 2 what
// pass 1's subtraction missed (h2 = V^T (w - V h)), and T takes h + h2; T is
// symmetric, and pass 1 wrote both of its entries.
template <int PASS>
__device__ __forceinline__ void put_dots(const EigArgs& a, int patch, int j, int warp, int lane) {
  double* T = a.T + (long long)patch * a.m * a.m;
  patch_sums(
      a.part, a.tile_begin[patch], a.tile_count[patch], a.mp1, j + 1, warp, lane,
      [&](int i) { return PASS == 2 ? T[i * a.m + j] : 0.0; },
      [&](int i, double s, double was) {
        a.hbuf[(long long)patch * a.mp1 + i] = s;
        const double h = PASS == 2 ? was + s : s;
        T[i * a.m + j] = h;
        T[j * a.m + i] = h;
      });
}

// ------------------------------------------------------------------ dots
// The groups of 8 basis vectors of a tile dealt over gridDim.y CTAs (the bits
// do not depend on how many).
template <int PASS>
__global__ void __launch_bounds__(kEigThreads, 2) ks_dots(EigArgs a, int j, const float* __restrict__ w) {
  const EigTile t = a.tiles[blockIdx.x];
  if (!a.active[t.patch]) return;
  const long long base = uniform(a.patches[t.patch].vec);
  uint32_t qv[kEigPix];
  float wv[kEigPix];
#pragma unroll
  for (int r = 0; r < kEigPix; r++) {
    const int p = t.p0 + threadIdx.x + r * kEigThreads;
    qv[r] = 4u * (uint32_t)(p < t.p1 ? p : t.p0);
    wv[r] = p < t.p1 ? ldu(w + base, qv[r]) : 0.f;
  }
  __shared__ float2 sred[kEigWarps * kRed];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  basis_dots(a, j, base, qv, wv, nullptr, sred, warp, lane, blockIdx.y, gridDim.y);
  cta_partials(sred, j + 1, a.part + (long long)blockIdx.x * a.mp1, blockIdx.y, gridDim.y);
  if (last_cta(a.counter + t.patch, a.tile_count[t.patch] * (int)gridDim.y)) put_dots<PASS>(a, t.patch, j, warp, lane);
}

// ------------------------------------------------------------------ SpMV
__global__ void __launch_bounds__(kEigThreads, 2) ks_spmv(EigArgs a, int j, const float* __restrict__ src,
                                                          int use_beta, float* __restrict__ dst) {
  const EigTile t = a.tiles[blockIdx.x];
  if (!a.active[t.patch]) return;
  const PatchDev P = a.patches[t.patch];
  // one thread forms the FP64 root and quotient; all wait for it at the barrier below
  __shared__ float inv_s;
  if (threadIdx.x == 0) inv_s = use_beta ? (float)(1.0 / sqrt(a.beta2[t.patch])) : 1.f;
  const long long base = uniform(P.vec);
  __shared__ int off[kUpper];
  if (threadIdx.x < kUpper) off[threadIdx.x] = c_up_dy[threadIdx.x] * P.W + c_up_dx[threadIdx.x];
  __syncthreads();
  // this thread's pixels; a pixel past the tile reads the tile's first one
  // (in bounds) and its results are dropped
  uint32_t qv[kEigPix];
  bool okv[kEigPix];
#pragma unroll
  for (int r = 0; r < kEigPix; r++) {
    const int p = t.p0 + threadIdx.x + r * kEigThreads;
    okv[r] = p < t.p1;
    qv[r] = 4u * (uint32_t)(okv[r] ? p : t.p0);
  }
  float acc[kEigPix];
#pragma unroll
  for (int r = 0; r < kEigPix; r++) acc[r] = 0.f;
#pragma unroll 2
  for (int k = 0; k < kUpper; k++) {
    const float* au = a.a_up + (long long)k * a.lvec + base;
    const float* xs = src + base;
    const int o = off[k];
    float cu[kEigPix], xu[kEigPix], cl[kEigPix], xl[kEigPix];
#pragma unroll
    for (int r = 0; r < kEigPix; r++) {
      const int q = (int)(qv[r] >> 2);
      cu[r] = au[q];
      xu[r] = xs[q + o];
      cl[r] = au[q - o];
      xl[r] = xs[q - o];
    }
#pragma unroll
    for (int r = 0; r < kEigPix; r++) {
      acc[r] = fmaf(cu[r], xu[r], acc[r]);
      acc[r] = fmaf(cl[r], xl[r], acc[r]);
    }
  }
  __syncthreads();
  const float inv = inv_s;
  float wv[kEigPix], xv[kEigPix];
#pragma unroll
  for (int r = 0; r < kEigPix; r++) {
    const float x = ldu(src + base, qv[r]) * inv;
    xv[r] = okv[r] ? x : 0.f;
    wv[r] = okv[r] ? fmaf(acc[r], inv, ldu(a.a_diag + base, qv[r]) * x) : 0.f;
  }
  float* Vj = a.V + (long long)j * a.lvec + base;
#pragma unroll
  for (int r = 0; r < kEigPix; r++) {
    if (!okv[r]) continue;
    stu(Vj, qv[r], xv[r]);
    stu(dst + base, qv[r], wv[r]);
  }
  // h_i = v_i . w for i <= j
  __shared__ float2 sred[kEigWarps * kRed];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  basis_dots(a, j, base, qv, wv, xv, sred, warp, lane);
  cta_partials(sred, j + 1, a.part + (long long)blockIdx.x * a.mp1);
  if (last_cta(a.counter + t.patch, a.tile_count[t.patch])) put_dots<1>(a, t.patch, j, warp, lane);
}

// w = A v_j and v_j alone: 256 pixels of a tile per CTA, one per thread.  A
// chain of load latencies on few tiles, so it is spread as wide as it goes:
// on one 321 x 481 image ks_mult + ks_dots take 8.7 + 11.8 us and
// ks_project + ks_dots 6.5 + 11.7 us, the whole step 52 us from 59.
__global__ void __launch_bounds__(kEigThreads) ks_mult(EigArgs a, int j, const float* __restrict__ src,
                                                       int use_beta, float* __restrict__ dst) {
  const EigTile t = a.tiles[blockIdx.x / kEigPix];
  if (!a.active[t.patch]) return;
  const int p0 = t.p0 + (int)(blockIdx.x % kEigPix) * kEigThreads, p = p0 + threadIdx.x;
  if (p0 >= t.p1) return;
  const PatchDev P = a.patches[t.patch];
  __shared__ int off[kUpper];
  __shared__ float inv_s;
  // one thread forms the FP64 root and quotient; all wait for it at the barrier
  if (threadIdx.x == kEigThreads - 1) inv_s = use_beta ? (float)(1.0 / sqrt(a.beta2[t.patch])) : 1.f;
  if (threadIdx.x < kUpper) off[threadIdx.x] = c_up_dy[threadIdx.x] * P.W + c_up_dx[threadIdx.x];
  __syncthreads();
  if (p >= t.p1) return;
  const long long q = P.vec + p;
  const float* au = a.a_up + q;
  const float* xs = src + q;
  float acc = 0.f;
  constexpr int NO = 8;  // offsets loaded together
  static_assert(kUpper % NO == 0, "offset groups");
#pragma unroll 1
  for (int k0 = 0; k0 < kUpper; k0 += NO, au += NO * a.lvec) {
    float cu[NO], xu[NO], cl[NO], xl[NO];
#pragma unroll
    for (int u = 0; u < NO; u++) {
      const int o = off[k0 + u];
      const float* al = au + u * a.lvec;
      cu[u] = al[0];
      xu[u] = xs[o];
      cl[u] = al[-o];
      xl[u] = xs[-o];
    }
#pragma unroll
    for (int u = 0; u < NO; u++) {
      acc = fmaf(cu[u], xu[u], acc);
      acc = fmaf(cl[u], xl[u], acc);
    }
  }
  const float inv = inv_s, x = xs[0] * inv;
  a.V[(long long)j * a.lvec + q] = x;
  dst[q] = fmaf(acc, inv, a.a_diag[q] * x);
}

// --------------------------------------------------------------- CGS pass
// MODE 1: w -= V h, then h2 = V^T w;  MODE 2: w -= V h2, then |w|^2.
// Pass 1 subtracts a projection of about |w|'s size (the cancellation of a
// converging step), so V h is formed in float-float and subtracted exactly;
// pass 2's V h2 is of rounding-error size and an FMA chain holds it.  Both
// sums run on pairs of pixels (f32x2).  Measured on one 321 x 481 image, whose
// basis stays in L2: 18.8 us (pass 1) and 9.1 us (pass 2) per launch, from
// 26.0 and 11.0 us with scalar sums, 64-bit addresses and a one-value-at-a-
// time tail; ks_restart 49 us from 117 us with one CTA per 2048 pixels.
template <int MODE>
__global__ void __launch_bounds__(kEigThreads, 2) ks_orth(EigArgs a, int j, float* __restrict__ w) {
  const EigTile t = a.tiles[blockIdx.x];
  if (!a.active[t.patch]) return;
  const PatchDev P = a.patches[t.patch];
  const long long base = uniform(P.vec);
  // projection coefficients as FP32 hi + lo pairs; the sum V h is formed in
  // float-float and subtracted from w before the single rounding to FP32, so
  // the cancellation of a converging step (|w - V h| << |w|) keeps its digits
  __shared__ float hs[kMaxKrylov + 1], hl[kMaxKrylov + 1];
  for (int i = threadIdx.x; i <= j; i += blockDim.x) {
    const double h = a.hbuf[(long long)t.patch * a.mp1 + i];
    hs[i] = (float)h;
    hl[i] = (float)(h - (double)hs[i]);
  }
  __syncthreads();
  uint32_t qv[kEigPix];
  bool okv[kEigPix];
  float wv[kEigPix];
  F2 sh[kEigPix / 2], sl[kEigPix / 2];  // pairs of pixels
#pragma unroll
  for (int r = 0; r < kEigPix; r++) {
    const int p = t.p0 + threadIdx.x + r * kEigThreads;
    okv[r] = p < t.p1;
    qv[r] = 4u * (uint32_t)(okv[r] ? p : t.p0);
    wv[r] = okv[r] ? ldu(w + base, qv[r]) : 0.f;
    sh[r / 2] = sl[r / 2] = f2(0.f, 0.f);
  }
  for (int i0 = 0; i0 <= j; i0 += kGrp) {
    float vv[kGrp][kEigPix];
#pragma unroll
    for (int u = 0; u < kGrp; u++) {
      const float* Vi = a.V + (long long)(i0 + u) * a.lvec + base;
#pragma unroll
      for (int r = 0; r < kEigPix; r++) vv[u][r] = (i0 + u <= j) ? ldu(Vi, qv[r]) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kGrp; u++) {
      if (i0 + u > j) break;
      const F2 h = f2(hs[i0 + u], hs[i0 + u]), h2 = f2(hl[i0 + u], hl[i0 + u]);
#pragma unroll
      for (int r = 0; r < kEigPix / 2; r++) {
        const F2 v = f2(vv[u][2 * r], vv[u][2 * r + 1]);
        if constexpr (MODE == 1) {
          ff_add_prod2(sh[r], sl[r], h, v);
          sl[r] = f2_fma(h2, v, sl[r]);
        } else {
          sh[r] = f2_fma(h, v, sh[r]);
        }
      }
    }
  }
#pragma unroll
  for (int r = 0; r < kEigPix; r++) {
    const float2 s2 = f2_split(sh[r / 2]), l2 = f2_split(sl[r / 2]);
    const float sr = r % 2 ? s2.y : s2.x, lr = r % 2 ? l2.y : l2.x;
    if constexpr (MODE == 1) {
      // w - (sr + lr) with the subtraction of sr exact (two-difference)
      const float d = wv[r] - sr;
      const float z = d - wv[r];
      const float e = (wv[r] - (d - z)) - (sr + z);
      wv[r] = okv[r] ? d + (e - lr) : 0.f;
    } else {
      wv[r] = okv[r] ? wv[r] - sr : 0.f;
    }
  }
#pragma unroll
  for (int r = 0; r < kEigPix; r++)
    if (okv[r]) stu(w + base, qv[r], wv[r]);
  __shared__ float2 sred[kEigWarps * kRed];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if constexpr (MODE == 1) {
    basis_dots(a, j, base, qv, wv, nullptr, sred, warp, lane);
    cta_partials(sred, j + 1, a.part + (long long)blockIdx.x * a.mp1);
  } else {
    float hi = 0.f, lo = 0.f;
#pragma unroll
    for (int r = 0; r < kEigPix; r++)
      if (okv[r]) ff_add_prod(hi, lo, wv[r], wv[r]);
    const float2 s = ff_warp_reduce(hi, lo);
    if (lane == 0) sred[warp * kRed] = s;
    cta_partials(sred, 1, a.part + (long long)blockIdx.x * a.mp1);
  }
  if (last_cta(a.counter + t.patch, a.tile_count[t.patch])) {
    if constexpr (MODE == 1) {
      put_dots<2>(a, t.patch, j, warp, lane);
    } else if (warp == 0) {
      double* T = a.T + (long long)t.patch * a.m * a.m;
      patch_sums(
          a.part, a.tile_begin[t.patch], a.tile_count[t.patch], a.mp1, 1, warp, lane, [](int) { return 0.0; },
          [&](int, double s, double) {
            if (!(s > 1e-60)) s = 1e-60;
            a.beta2[t.patch] = s;
            if (j + 1 < a.m) {
              const double b = sqrt(s);
              T[(j + 1) * a.m + j] = b;
              T[j * a.m + (j + 1)] = b;
            }
          });
    }
  }
}

// w -= V h alone, as ks_orth<1> does it: 512 pixels per CTA, two per thread
constexpr int kProjPix = 2, kProjSplit = kEigPix / kProjPix;
__global__ void __launch_bounds__(kEigThreads) ks_project(EigArgs a, int j, float* __restrict__ w) {
  const EigTile t = a.tiles[blockIdx.x / kProjSplit];
  if (!a.active[t.patch]) return;
  const int p0 = t.p0 + (int)(blockIdx.x % kProjSplit) * kProjPix * kEigThreads;
  if (p0 >= t.p1) return;
  const PatchDev P = a.patches[t.patch];
  const long long base = uniform(P.vec);
  __shared__ float hs[kMaxKrylov + 1], hl[kMaxKrylov + 1];
  for (int i = threadIdx.x; i <= j; i += blockDim.x) {
    const double h = a.hbuf[(long long)t.patch * a.mp1 + i];
    hs[i] = (float)h;
    hl[i] = (float)(h - (double)hs[i]);
  }
  __syncthreads();
  const int pa = p0 + threadIdx.x, pb = pa + kEigThreads;
  const uint32_t qa = 4u * (uint32_t)(pa < t.p1 ? pa : t.p0), qb = 4u * (uint32_t)(pb < t.p1 ? pb : t.p0);
  const float wv[2] = {ldu(w + base, qa), ldu(w + base, qb)};
  F2 sh = f2(0.f, 0.f), sl = sh;
  constexpr int NV = 16;  // basis vectors loaded together
  for (int i0 = 0; i0 <= j; i0 += NV) {
    F2 vv[NV];
#pragma unroll
    for (int u = 0; u < NV; u++) {
      const float* Vi = a.V + (long long)(i0 + u) * a.lvec + base;
      vv[u] = i0 + u <= j ? f2(ldu(Vi, qa), ldu(Vi, qb)) : f2(0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < NV; u++) {
      if (i0 + u > j) break;
      ff_add_prod2(sh, sl, f2(hs[i0 + u], hs[i0 + u]), vv[u]);
      sl = f2_fma(f2(hl[i0 + u], hl[i0 + u]), vv[u], sl);
    }
  }
  const float2 s2 = f2_split(sh), l2 = f2_split(sl);
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const float sr = r ? s2.y : s2.x, lr = r ? l2.y : l2.x;
    const float d = wv[r] - sr;
    const float z = d - wv[r];
    const float e = (wv[r] - (d - z)) - (sr + z);
    if ((r ? pb : pa) < t.p1) stu(w + base, r ? qb : qa, d + (e - lr));
  }
}

// -------------------------------------------------------------- restart
// Vout[:, 0..nk) = V[:, 0..m) Y[:, 0..nk) per pixel, then Vout[nk] = w / beta
// (restart, Vout is the other basis buffer) -- or, for a converged patch
// (FINAL), the nk = nvec Ritz vectors into evec_out.  A CTA per 256 pixels: a
// restart is one launch between host round trips, so it is spread as wide as
// it goes.
// Y is split into FP32 hi + lo; the hi products are summed by FMA in groups of
// four folded into a float-float by TwoSum, the lo products into the low word:
// an FMA chain's rounding (about sqrt(m) units) would show in the residuals
// and, at a restart, in the relation that their estimate relies on.  A thread
// takes one pixel and 16 outputs per pass over V, so each basis value is loaded
// once per pass and each 16-byte broadcast of Y (shared memory, zero-padded)
// feeds 4 FMAs.
template <bool FINAL>
__global__ void __launch_bounds__(kEigThreads, 2) ks_restart(EigArgs a, const float* __restrict__ w,
                                                            float* __restrict__ vout,
                                                            float* __restrict__ evec_out) {
  constexpr int COLS = 16;  // outputs per pass over V
  const EigTile t = a.tiles[blockIdx.x / kEigPix];
  const int mode = a.decision[t.patch];  // 0 idle, 1 restart, 2 final
  if (mode != (FINAL ? 2 : 1)) return;
  const PatchDev P = a.patches[t.patch];
  const int nk = a.nkeep[t.patch], m = a.m;
  extern __shared__ float4 ysh4[];  // [m][COLS / 4] hi, then (FINAL) lo
  float* ysh = (float*)ysh4;
  const double* Y = a.Y + (long long)t.patch * m * m;
  const int base = (int)P.vec;
  // 256 pixels of the tile per CTA
  const int p0 = t.p0 + (int)(blockIdx.x % kEigPix) * kEigThreads, p = p0 + threadIdx.x;
  if (p0 >= t.p1) return;
  float* out = FINAL ? evec_out : vout;
  for (int c0 = 0; c0 < nk; c0 += COLS) {
    __syncthreads();
    for (int idx = threadIdx.x; idx < m * COLS; idx += blockDim.x) {
      const int i = idx / COLS, c = c0 + idx % COLS;
      const double y = c < nk ? Y[i * m + c] : 0.0;
      const float yh = (float)y;
      ysh[idx] = yh;
      ysh[m * COLS + idx] = (float)(y - (double)yh);
    }
    __syncthreads();
    if (p < t.p1) {
      const int q = base + p;
      float acc[COLS], lo[COLS], g[COLS];
#pragma unroll
      for (int c = 0; c < COLS; c++) acc[c] = lo[c] = g[c] = 0.f;
#pragma unroll 8
      for (int i = 0; i < m; i++) {
        const float v = a.V[(long long)i * a.lvec + q];
#pragma unroll
        for (int c4 = 0; c4 < COLS / 4; c4++) {
          const float4 y = ysh4[i * (COLS / 4) + c4];
          const float yv[4] = {y.x, y.y, y.z, y.w};
          const float4 yl = ysh4[(m + i) * (COLS / 4) + c4];
          const float ylv[4] = {yl.x, yl.y, yl.z, yl.w};
#pragma unroll
          for (int j = 0; j < 4; j++) {
            g[4 * c4 + j] = fmaf(yv[j], v, g[4 * c4 + j]);
            lo[4 * c4 + j] = fmaf(ylv[j], v, lo[4 * c4 + j]);
          }
        }
        if ((i & 3) == 3 || i == m - 1) {
#pragma unroll
          for (int c = 0; c < COLS; c++) {
            const float sum = acc[c] + g[c], z = sum - acc[c];
            lo[c] += (acc[c] - (sum - z)) + (g[c] - z);
            acc[c] = sum;
            g[c] = 0.f;
          }
        }
      }
#pragma unroll
      for (int c = 0; c < COLS; c++)
        if (c0 + c < nk) out[(long long)(c0 + c) * a.lvec + q] = acc[c] + lo[c];
    }
  }
  if constexpr (!FINAL) {
    const float inv = (float)(1.0 / sqrt(a.beta2[t.patch]));
    if (p < t.p1) vout[(long long)nk * a.lvec + base + p] = w[base + p] * inv;
  }
}

// start vector: a fixed hash per pixel, |w|^2 into beta2 (through the same
// last-CTA reduction)
__device__ __forceinline__ float hash_unit(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352dU;
  x ^= x >> 15;
  x *= 0x846ca68bU;
  x ^= x >> 16;
  return (float)(x & 0xffffff) * (1.0f / 16777216.0f) - 0.5f;
}

__global__ void __launch_bounds__(kEigThreads) ks_init(EigArgs a, float* __restrict__ w) {
  const EigTile t = a.tiles[blockIdx.x];
  if (!a.active[t.patch]) return;
  const PatchDev P = a.patches[t.patch];
  float hi = 0.f, lo = 0.f;
  for (int r = 0; r < kEigPix; r++) {
    const int p = t.p0 + threadIdx.x + r * kEigThreads;
    if (p >= t.p1) continue;
    const float v = hash_unit((uint32_t)p * 2654435761u + 12345u);
    w[P.vec + p] = v;
    ff_add_prod(hi, lo, v, v);
  }
  __shared__ float2 sred[kEigWarps * kRed];
  const float2 s = ff_warp_reduce(hi, lo);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) sred[warp * kRed] = s;
  cta_partials(sred, 1, a.part + (long long)blockIdx.x * a.mp1);
  if (last_cta(a.counter + t.patch, a.tile_count[t.patch]) && warp == 0) {
    const int tb = a.tile_begin[t.patch], tc = a.tile_count[t.patch];
    patch_sums(
        a.part, tb, tc, a.mp1, 1, warp, lane, [](int) { return 0.0; },
        [&](int, double s2, double) { a.beta2[t.patch] = s2; });
  }
}

cudaError_t ks_launch_init(const EigArgs& a, int ntiles, float* w, cudaStream_t s) {
  ks_init<<<ntiles, kEigThreads, 0, s>>>(a, w);
  return cudaGetLastError();
}
// CTAs per tile of the dots: two waves of the 304 that the 152 SMs hold
static int dot_split(int ntiles, int j) { return std::min(j / kGrp + 1, std::max(1, 608 / ntiles)); }

cudaError_t ks_launch_spmv(const EigArgs& a, int ntiles, int j, const float* src, int use_beta,
                           float* dst, cudaStream_t s) {
  if (ntiles > kEigSplitTiles) {
    ks_spmv<<<ntiles, kEigThreads, 0, s>>>(a, j, src, use_beta, dst);
  } else {
    ks_mult<<<ntiles * kEigPix, kEigThreads, 0, s>>>(a, j, src, use_beta, dst);
    ks_dots<1><<<dim3(ntiles, dot_split(ntiles, j)), kEigThreads, 0, s>>>(a, j, dst);
  }
  return cudaGetLastError();
}
cudaError_t ks_launch_orth(const EigArgs& a, int ntiles, int j, int mode, float* w, cudaStream_t s) {
  if (mode == 2) {
    ks_orth<2><<<ntiles, kEigThreads, 0, s>>>(a, j, w);
  } else if (ntiles > kEigSplitTiles) {
    ks_orth<1><<<ntiles, kEigThreads, 0, s>>>(a, j, w);
  } else {
    ks_project<<<ntiles * kProjSplit, kEigThreads, 0, s>>>(a, j, w);
    ks_dots<2><<<dim3(ntiles, dot_split(ntiles, j)), kEigThreads, 0, s>>>(a, j, w);
  }
  return cudaGetLastError();
}
cudaError_t ks_launch_restart(const EigArgs& a, int ntiles, const float* w, float* vout, float* evec,
                              cudaStream_t s, bool any_restart, bool any_final) {
  if (any_restart) ks_restart<false><<<ntiles * kEigPix, kEigThreads, 2 * a.m * 16 * sizeof(float), s>>>(a, w, vout, evec);
  if (any_final) ks_restart<true><<<ntiles * kEigPix, kEigThreads, 2 * a.m * 16 * sizeof(float), s>>>(a, w, vout, evec);
  return cudaGetLastError();
}

}  // namespace gpb
