// k_stitch.cu -- whole-image gPb planes from the last batch's halo'd patches,
// on the device (replaces Pieces2Gpb, src/utilities.cpp:180-213, which
// copies every part's full box into the image in loop order so that later
// parts overwrite the overlaps).
//
// One launch gathers: a CTA owns a 32 x 32 tile of the image, finds the boxes
// that touch it (256 at a time, in patch order) and each thread takes its
// pixels' values from them.  The CTAs cover the tiles around all boxes, or,
// where the boxes are scattered and that would be more, each box's own tiles
// (see launch_stitch).
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

#include <algorithm>
#include <vector>

#include "gpb_internal.h"
#include "kernels.h"

namespace gpb {

namespace {

// boxes passed in the launch itself: no buffer, no copy
struct StitchFew {
  StitchSpan b[kStitchFew];
};

constexpr int ST_T = 32, ST_ROWS = 4;  // tile side; rows per thread, 8 apart

__device__ __forceinline__ float patch_orient(const float* orient, const PatchDev& P, int colmajor, int o, int y,
                                              int x) {
  const long long base = 8 * P.pix + (long long)o * P.N;
  return orient[base + (colmajor ? (long long)x * P.H + y : (long long)y * P.W + x)];
}

// weight of patch pixel (y, x): 1 in the interior, falling linearly to
// 1 / (2 ramp) at a patch edge that lies inside the image
__device__ __forceinline__ float stitch_weight(const StitchSpan& b, const PatchDev& P, int y, int x, int img_w,
                                               int img_h, float ramp) {
  float w = 1.f;
  if (b.oy > 0) w = fminf(w, (y + 0.5f) / ramp);
  if (b.ox > 0) w = fminf(w, (x + 0.5f) / ramp);
  if (b.oy + P.H < img_h) w = fminf(w, (P.H - y - 0.5f) / ramp);
  if (b.ox + P.W < img_w) w = fminf(w, (P.W - x - 0.5f) / ramp);
  return w;
}

// a rectangle of tiles, cols wide
struct StitchGrid {
  unsigned x0, y0, cols;
};
// the tiles [x0, x1) x [y0, y1) that a box touches; none if it is empty
struct TileRange {
  unsigned x0, x1, y0, y1;
};
__host__ __device__ __forceinline__ TileRange span_tiles(const StitchSpan& b) {
  return {b.x0 / ST_T, (b.x1 + ST_T - 1) / ST_T, b.y0 / ST_T, (b.y1 + ST_T - 1) / ST_T};
}

// A CTA's tile is that of its place in `grid`, or (OWN) of its place in the
// tiles of the last box whose `first` is at most its number.
template <bool BLEND, bool OWN>
__global__ void __launch_bounds__(256) k_stitch(const PatchDev* __restrict__ patches,
                                                const __grid_constant__ StitchFew few,
                                                const StitchSpan* __restrict__ many, int n, StitchGrid grid,
                                                const float* __restrict__ nmax, const float* __restrict__ orient,
                                                int colmajor, int img_w, int img_h, float ramp,
                                                float* __restrict__ out_nmax, float* __restrict__ out_orient) {
  __shared__ int list[256], warp_n[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const StitchSpan* boxes = many ? many : few.b;
  unsigned tx, ty;
  int own = 0;  // the box whose tiles these are
  if constexpr (!OWN) {
    tx = grid.x0 + blockIdx.x % grid.cols;
    ty = grid.y0 + blockIdx.x / grid.cols;
  } else {
    int hi = n;  // boxes without tiles share their successor's `first`
    while (hi - own > 1) {
      const int mid = own + (hi - own) / 2;
      if (boxes[mid].first <= blockIdx.x) own = mid;
      else hi = mid;
    }
    const TileRange r = span_tiles(boxes[own]);
    const unsigned t = blockIdx.x - boxes[own].first;
    tx = r.x0 + t % (r.x1 - r.x0);
    ty = r.y0 + t / (r.x1 - r.x0);
  }
  const unsigned gx = tx * ST_T + lane, gy0 = ty * ST_T + warp;  // images end below 2^31
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
      const TileRange r = span_tiles(boxes[p0 + threadIdx.x]);
      hit = tx >= r.x0 && tx < r.x1 && ty >= r.y0 && ty < r.y1;
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
    // a tile that several boxes share belongs to the first of them
    if constexpr (OWN) {
      if (own >= 0 && total > 0) {
        if (list[0] != own) return;
        own = -1;
      }
    }
    for (int i = 0; i < total; i++) {
      const int pi = list[i];
      const StitchSpan b = boxes[pi];
      const PatchDev P = patches[pi];
      if (gx < b.x0 || gx >= b.x1) continue;
      const int x = (int)gx - b.ox;  // patch coordinates
#pragma unroll
      for (int k = 0; k < ST_ROWS; k++) {
        const unsigned gy = gy0 + 8 * k;
        if (gy < b.y0 || gy >= b.y1) continue;
        const int y = (int)gy - b.oy;
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
#pragma unroll
  for (int k = 0; k < ST_ROWS; k++) {
    const unsigned gy = gy0 + 8 * k;  // inside the image where a box covers it
    const long long g = (long long)gy * img_w + gx;
    if constexpr (BLEND) {
      if (!(acc[k][0] > 0.f)) continue;
      const float r = 1.f / acc[k][0];
      out_nmax[g] = acc[k][1] * r;
#pragma unroll
      for (int o = 0; o < 8; o++) out_orient[o * plane + g] = acc[k][2 + o] * r;
    } else {
      if (win[k] < 0) continue;
      const StitchSpan b = boxes[win[k]];
      const PatchDev P = patches[win[k]];
      const int y = (int)gy - b.oy, x = (int)gx - b.ox;
      out_nmax[g] = nmax[P.pix + (long long)y * P.W + x];
#pragma unroll
      for (int o = 0; o < 8; o++) out_orient[o * plane + g] = patch_orient(orient, P, colmajor, o, y, x);
    }
  }
}

}  // namespace

cudaError_t launch_stitch(const PatchDev* patches, const StitchBox* boxes, StitchSpan* dev_spans, int n, bool blend,
                          const float* nmax, const float* orient, int colmajor, int img_w, int img_h, float ramp,
                          float* out_nmax, float* out_orient, cudaStream_t s) {
  // A stitch may fill a small part of a large image (the last batch's), so the
  // CTAs follow the boxes, not the image: one per tile of the rectangle around
  // them, or one per tile of each box where those are fewer.  Boxes that tile
  // the image leave nothing between them and share their edge tiles, so there
  // the rectangle is smaller (16 boxes of 266^2 in 1024^2: 1024 CTAs against
  // 1444).  Measured, a box of 256^2 in an image of 8192^2: 3.4 us, 65 us with a
  // CTA for every tile of the image; 16 of them scattered over it: 12 against
  // 69 us (blended 20 against 153).
  StitchFew few = {};
  std::vector<StitchSpan> many(dev_spans ? n : 0);
  StitchSpan* spans = dev_spans ? many.data() : few.b;
  auto clip = [](long long v, int lim) { return (unsigned)std::min(std::max(v, 0LL), (long long)std::max(lim, 0)); };
  long long own = 0;
  TileRange all = {0xffffffffu, 0, 0xffffffffu, 0};
  for (int i = 0; i < n; i++) {
    const StitchBox& b = boxes[i];
    const long long x = (long long)b.ox + b.x, y = (long long)b.oy + b.y;
    StitchSpan& p = spans[i];
    p = {b.ox, b.oy, clip(x, img_w), clip(y, img_h), clip(x + b.w, img_w), clip(y + b.h, img_h), (unsigned)own};
    if (p.x0 >= p.x1 || p.y0 >= p.y1) {
      p.x0 = p.x1 = p.y0 = p.y1 = 0;  // covers nothing
      continue;
    }
    const TileRange r = span_tiles(p);
    own += (long long)(r.x1 - r.x0) * (r.y1 - r.y0);
    all = {std::min(all.x0, r.x0), std::max(all.x1, r.x1), std::min(all.y0, r.y0), std::max(all.y1, r.y1)};
  }
  if (own == 0) return cudaSuccess;
  const long long around = (long long)(all.x1 - all.x0) * (all.y1 - all.y0), ctas = std::min(around, own);
  if (ctas > 0x7fffffffLL) return cudaErrorInvalidValue;  // 2^41 pixels
  const StitchGrid grid = {all.x0, all.y0, all.x1 - all.x0};
  if (dev_spans) {
    const cudaError_t e = cudaMemcpyAsync(dev_spans, spans, n * sizeof(StitchSpan), cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) return e;
  }
  auto* kernel = around <= own ? (blend ? k_stitch<true, false> : k_stitch<false, false>)
                               : (blend ? k_stitch<true, true> : k_stitch<false, true>);
  kernel<<<(unsigned)ctas, 256, 0, s>>>(patches, few, dev_spans, n, grid, nmax, orient, colmajor, img_w, img_h, ramp,
                                        out_nmax, out_orient);
  return cudaGetLastError();
}

}  // namespace gpb
