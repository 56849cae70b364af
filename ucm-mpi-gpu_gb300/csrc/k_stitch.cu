// k_stitch.cu -- whole-image gPb planes from the last batch's halo'd patches,
// on the device (replaces Pieces2Gpb, src/utilities.cpp:180-213, which
// copies every part's full box into the image in loop order so that later
// parts overwrite the overlaps).
//
// One launch gathers: a CTA owns a 32 x 32 tile of the image, finds the boxes
// that touch it (256 at a time, in patch order) and each thread takes its
// pixels' values from them.
//   LAST, INTERIOR  the last patch whose box (its whole box, or its interior)
//                   covers the pixel
//   BLEND           sum of weight * value over sum of weight, in patch order;
//                   weights fall linearly over the overlap
// A pixel that no box covers is left as it was.  Bound by HBM (36 bytes read
// per covering patch and 36 written per pixel) and, at 1024^2, by the launch:
// 17 us there (16 patches), a whole call 43 us, from 138 us with a launch per
// patch, atomics into a zeroed 10-plane accumulator and a normalising pass.
//
// Patch values are read in the context's compat layout (orient planes
// row-major for GPB_COMPAT_CPU, column-major for GPB_COMPAT_DAMASCENE); the
// image planes are row-major, in the patch output's plane order.
#include <stdint.h>

#include "gpb_internal.h"
#include "kernels.h"

namespace gpb {

namespace {

// boxes passed in the launch itself: no buffer, no copy
struct StitchFew {
  StitchBox b[kStitchFew];
};

constexpr int ST_T = 32, ST_ROWS = 4;  // tile side; rows per thread, 8 apart

__device__ __forceinline__ float patch_orient(const float* orient, const PatchDev& P, int colmajor, int o, int y,
                                              int x) {
  const long long base = 8 * P.pix + (long long)o * P.N;
  return orient[base + (colmajor ? (long long)x * P.H + y : (long long)y * P.W + x)];
}

// weight of patch pixel (y, x): 1 in the interior, falling linearly to
// 1 / (2 ramp) at a patch edge that lies inside the image
__device__ __forceinline__ float stitch_weight(const StitchBox& b, const PatchDev& P, int y, int x, int img_w,
                                               int img_h, float ramp) {
  float w = 1.f;
  if (b.oy > 0) w = fminf(w, (y + 0.5f) / ramp);
  if (b.ox > 0) w = fminf(w, (x + 0.5f) / ramp);
  if (b.oy + P.H < img_h) w = fminf(w, (P.H - y - 0.5f) / ramp);
  if (b.ox + P.W < img_w) w = fminf(w, (P.W - x - 0.5f) / ramp);
  return w;
}

template <bool BLEND>
__global__ void __launch_bounds__(256) k_stitch(const PatchDev* __restrict__ patches,
                                                const __grid_constant__ StitchFew few,
                                                const StitchBox* __restrict__ many, int n, unsigned cols,
                                                const float* __restrict__ nmax, const float* __restrict__ orient,
                                                int colmajor, int img_w, int img_h, float ramp,
                                                float* __restrict__ out_nmax, float* __restrict__ out_orient) {
  __shared__ int list[256], warp_n[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const StitchBox* boxes = many ? many : few.b;
  const int tx0 = (int)(blockIdx.x % cols) * ST_T, ty0 = (int)(blockIdx.x / cols) * ST_T;
  const int gx = tx0 + lane;
  const long long plane = (long long)img_w * img_h;
  int win[ST_ROWS];           // the last covering patch
  float acc[ST_ROWS][10];     // weight, then weight * value of the planes
#pragma unroll
  for (int k = 0; k < ST_ROWS; k++) {
    win[k] = -1;
#pragma unroll
    for (int c = 0; c < 10; c++) acc[k][c] = 0.f;
  }
  for (int p0 = 0; p0 < n; p0 += 256) {
    // the boxes of this run that touch the tile, in order
    bool hit = false;
    if (p0 + (int)threadIdx.x < n) {
      const StitchBox b = boxes[p0 + threadIdx.x];
      const long long x0 = (long long)b.ox + b.x, y0 = (long long)b.oy + b.y;
      hit = x0 < tx0 + ST_T && x0 + b.w > tx0 && y0 < ty0 + ST_T && y0 + b.h > ty0;
    }
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (lane == 0) warp_n[warp] = __popc(m);
    __syncthreads();
    int at = 0, total = 0;
#pragma unroll
    for (int w = 0; w < 8; w++) {
      if (w < warp) at += warp_n[w];
      total += warp_n[w];
    }
    if (hit) list[at + __popc(m & ((1u << lane) - 1u))] = p0 + threadIdx.x;
    __syncthreads();
    for (int i = 0; i < total; i++) {
      const int pi = list[i];
      const StitchBox b = boxes[pi];
      const PatchDev P = patches[pi];
      const int x = gx - b.ox;  // patch coordinates
      if (x < b.x || x >= b.x + b.w) continue;
#pragma unroll
      for (int k = 0; k < ST_ROWS; k++) {
        const int y = ty0 + warp + 8 * k - b.oy;
        if (y < b.y || y >= b.y + b.h) continue;
        if constexpr (BLEND) {
          const float w = stitch_weight(b, P, y, x, img_w, img_h, ramp);
          acc[k][0] = __fadd_rn(acc[k][0], w);
          acc[k][1] = __fadd_rn(acc[k][1], __fmul_rn(w, nmax[P.pix + (long long)y * P.W + x]));
#pragma unroll
          for (int o = 0; o < 8; o++)
            acc[k][2 + o] = __fadd_rn(acc[k][2 + o], __fmul_rn(w, patch_orient(orient, P, colmajor, o, y, x)));
        } else {
          win[k] = pi;
        }
      }
    }
    __syncthreads();
  }
  if (gx >= img_w) return;
#pragma unroll
  for (int k = 0; k < ST_ROWS; k++) {
    const int gy = ty0 + warp + 8 * k;
    if (gy >= img_h) continue;
    const long long g = (long long)gy * img_w + gx;
    if constexpr (BLEND) {
      if (!(acc[k][0] > 0.f)) continue;
      const float r = 1.f / acc[k][0];
      out_nmax[g] = acc[k][1] * r;
#pragma unroll
      for (int o = 0; o < 8; o++) out_orient[o * plane + g] = acc[k][2 + o] * r;
    } else {
      if (win[k] < 0) continue;
      const StitchBox b = boxes[win[k]];
      const PatchDev P = patches[win[k]];
      const int y = gy - b.oy, x = gx - b.ox;
      out_nmax[g] = nmax[P.pix + (long long)y * P.W + x];
#pragma unroll
      for (int o = 0; o < 8; o++) out_orient[o * plane + g] = patch_orient(orient, P, colmajor, o, y, x);
    }
  }
}

}  // namespace

cudaError_t launch_stitch(const PatchDev* patches, const StitchBox* host_boxes, const StitchBox* boxes, int n,
                          bool blend, const float* nmax, const float* orient, int colmajor, int img_w, int img_h,
                          float ramp, float* out_nmax, float* out_orient, cudaStream_t s) {
  StitchFew few = {};
  if (!boxes)
    for (int i = 0; i < n; i++) few.b[i] = host_boxes[i];
  const unsigned cols = (unsigned)((img_w + (long long)ST_T - 1) / ST_T);
  const long long tiles = cols * ((img_h + (long long)ST_T - 1) / ST_T);
  if (tiles > 0x7fffffffLL) return cudaErrorInvalidValue;  // planes of 2^41 pixels
  if (blend)
    k_stitch<true><<<(unsigned)tiles, 256, 0, s>>>(patches, few, boxes, n, cols, nmax, orient, colmajor, img_w, img_h,
                                                   ramp, out_nmax, out_orient);
  else
    k_stitch<false><<<(unsigned)tiles, 256, 0, s>>>(patches, few, boxes, n, cols, nmax, orient, colmajor, img_w, img_h,
                                                    ramp, out_nmax, out_orient);
  return cudaGetLastError();
}

}  // namespace gpb
