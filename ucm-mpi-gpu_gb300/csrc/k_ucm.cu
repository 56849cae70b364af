// k_ucm.cu -- the data-parallel stages of the oriented watershed transform
// and the ultrametric contour map (Contours2Ucm, src/contours2ucm.cpp).
//
//   k_ucm_pbmax    max over the 8 orientation planes, per-image min / max
//                  (contours2ucm.cpp:255-270)
//   k_ucm_quant    8-bit quantisation, FP64 alpha/beta and round-half-even
//                  saturation as OpenCV's convertTo (contours2ucm.cpp:272-278)
//   k_ws_rowsort   per row, the columns stably sorted by grey level
//   k_ws_flood     the level-by-level, raster-order flooding of
//                  watershed_yupeng (src/watershed.cpp:28-108) as a wavefront:
//                  level l of row x is processed at step t = 2l + x, when
//                  every pixel it reads (rows x-1..x+1 at lower levels, row
//                  x-1 at the same level, its own row to the left) is final
//                  and no other thread of the step writes a row it reads
//   k_ucm_paint    contour-strength painting along the fitted edges
//                  (contours2ucm.cpp:374-399)
//   k_ucm_super    SuperContour4C (contours2ucm.cpp:24-78) on the doubled grid
//   k_art_*        CleanWatersheds (contours2ucm.cpp:80-189): isolated zeros
//                  of the doubled grid, fixed in row-major order
//   k_ccl_*        8-connected labelling of the zeros of the cleaned grid,
//                  numbered in row-major order of each component's first
//                  cell (bwlabelManu, src/MATLAB_functions.cpp:164-217)
//   k_ucm_finish   region labels of the pixels and the padded strength grid
//                  ws_wt2 (contours2ucm.cpp:439-458)
//
// Every launch covers all images of a batch, each with CTAs in proportion to
// its size (UcmPart), except the flooding, the small scans (one CTA per image)
// and the artefact fixes (one thread per image).
#include <stdint.h>

#include <algorithm>

#include "ucm_dev.h"

namespace gpb {

namespace {

__device__ __forceinline__ unsigned f2ord(float f) {  // order-preserving float -> uint
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

}  // namespace

// the images of a launch and the kind of its CTAs
struct UcmLaunch {
  const UcmView* __restrict__ views;
  int n;
  UcmKind kind;
};
// this CTA's image, its number among the image's CTAs and how many those are
struct UcmPart {
  const UcmView& V;
  int cta, ctas;
};
// MUL: CTAs per counted one.  Whole warps, before any thread has left: a search
// by 32 places at a time, one load up to 32 images.
template <int MUL = 1>
__device__ __forceinline__ UcmPart ucm_part(const UcmLaunch& l) {
  const int b = (int)(blockIdx.x / MUL), lane = threadIdx.x & 31;
  int lo = 0, hi = l.n;  // first of lo <= b < first of hi
  while (hi - lo > 1) {
    const int step = (hi - lo + 31) / 32, i = lo + lane * step;
    const unsigned m = __ballot_sync(0xffffffffu, i < hi && l.views[i].first[l.kind] <= b);
    lo += (__popc(m) - 1) * step;
    hi = min(hi, lo + step);
  }
  const int f = l.views[lo].first[l.kind] * MUL;
  return {l.views[lo], (int)blockIdx.x - f, l.views[lo + 1].first[l.kind] * MUL - f};
}

// ---------------------------------------------------------------- pb, u8

__global__ void __launch_bounds__(256) k_ucm_pbmax(UcmLaunch l) {
  const UcmPart me = ucm_part(l);
  const UcmView& V = me.V;
  const float* __restrict__ orient = V.orient;
  const long long N = (long long)V.H * V.W;
  float* __restrict__ pb = V.s.pb;
  unsigned* mm = V.s.mm;
  if ((long long)me.cta * blockDim.x >= N) return;
  unsigned lo = 0xffffffffu, hi = 0u;
  for (long long i = (long long)me.cta * blockDim.x + threadIdx.x; i < N; i += (long long)me.ctas * blockDim.x) {
    float m = orient[i];
    for (int o = 1; o < 8; o++) {
      const float v = orient[(long long)o * N + i];
      if (m < v) m = v;  // the later plane wins only when strictly larger
    }
    pb[i] = m;
    lo = min(lo, f2ord(m));
    hi = max(hi, f2ord(m));
  }
  for (int d = 16; d; d >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, d));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, d));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMax(mm, ~lo);  // both start at 0
    atomicMax(mm + 1, hi);
  }
}

__global__ void __launch_bounds__(256) k_ucm_quant(UcmLaunch l) {
  const UcmPart me = ucm_part(l);
  const UcmView& V = me.V;
  const float* __restrict__ pb = V.s.pb;
  uint8_t* __restrict__ q = V.s.q;
  const long long N = (long long)V.H * V.W;
  const unsigned* mm = V.s.mm;
  const double lo = (double)ord2f(~mm[0]), hi = (double)ord2f(mm[1]);
  const double alpha = 255.0 / (hi - lo), beta = __ddiv_rn(-255.0 * lo, hi - lo);
  for (long long i = (long long)me.cta * blockDim.x + threadIdx.x; i < N; i += (long long)me.ctas * blockDim.x) {
    const double v = __dadd_rn(__dmul_rn((double)pb[i], alpha), beta);
    uint8_t r = 0;
    if (v == v) {  // NaN (a constant image) saturates to 0
      const double t = rint(v);
      r = (uint8_t)(t < 0.0 ? 0.0 : (t > 255.0 ? 255.0 : t));
    }
    q[i] = r;
  }
}

// ---------------------------------------------------------------- flooding

// One warp per row: a stable counting sort of the row's columns by level.  The
// levels are read with __ldg, so that the loads may pass the warp's barriers
// (60,000 columns: 662 us, 1057 without).
// off[row * 257 + l] is the first position of level l; cols[row * W + k]
// the k-th column in (level, column) order.
__global__ void __launch_bounds__(32) k_ws_rowsort(UcmLaunch l) {
  const UcmPart me = ucm_part(l);
  const UcmView& V = me.V;
  const uint8_t* __restrict__ q = V.s.q;
  const int H = V.H, W = V.W;
  int32_t* __restrict__ off = V.s.off;
  uint16_t* __restrict__ cols = V.s.cols;
  __shared__ int cnt[256];
  const int row = me.cta, lane = threadIdx.x;
  if (row >= H) return;
  for (int v = lane; v < 256; v += 32) cnt[v] = 0;
  __syncwarp();
  const uint8_t* r = q + (size_t)row * W;
  const unsigned lt = (1u << lane) - 1u;
  for (int c0 = 0; c0 < W; c0 += 32) {
    const int c = c0 + lane;
    const bool in = c < W;
    const int v = in ? __ldg(r + c) : 256 + lane;  // out-of-row lanes match nobody
    const unsigned peers = __match_any_sync(0xffffffffu, v);
    if (in && (peers & lt) == 0) cnt[v] += __popc(peers);
    __syncwarp();
  }
  // exclusive scan of the 256 counts: 8 per lane
  int loc[8], s = 0;
  for (int k = 0; k < 8; k++) {
    loc[k] = s;
    s += cnt[lane * 8 + k];
  }
  int inc = s;
  for (int d = 1; d < 32; d <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc += t;
  }
  const int base = inc - s;
  __syncwarp();
  for (int k = 0; k < 8; k++) {
    cnt[lane * 8 + k] = base + loc[k];
    off[(size_t)row * 257 + lane * 8 + k] = base + loc[k];
  }
  if (lane == 0) off[(size_t)row * 257 + 256] = W;
  __syncwarp();
  for (int c0 = 0; c0 < W; c0 += 32) {
    const int c = c0 + lane;
    const bool in = c < W;
    const int v = in ? __ldg(r + c) : 256 + lane;
    const unsigned peers = __match_any_sync(0xffffffffu, v);
    if (in) cols[(size_t)row * W + cnt[v] + __popc(peers & lt)] = (uint16_t)c;
    __syncwarp();
    if (in && (peers & lt) == 0) cnt[v] += __popc(peers);
    __syncwarp();
  }
}

// One CTA of 1024 threads per image; warp w owns grey levels w, w + 32, ...
// At step t a warp takes, level by level, the row t - 2l of its level l
// and walks that row's pixels of level l in column order, 32 at a time:
// every lane gathers the labels of its pixel's 8 neighbours at once, then
// runs of adjacent pixels are resolved lane by lane, and most lanes settle
// without waiting because their label cannot depend on the left one.  The
// next 32 pixels' neighbours are loaded before the current ones resolve;
// the one of them that the current 32 may still write (the left neighbour
// of the next first pixel) is taken from the current last pixel instead.
// ws is -1 (not reached), 0 (watershed pixel) or a region label (> 0): a
// new region takes the label 1 + its pixel index.  It has a border of one
// pixel that stays -1, so the gathers need no bounds checks.
// Bound by the chain of 255 x 2 + H steps on the image's one SM: it issues in
// a third of its cycles (321 x 481: 6.3 M instructions, 34 %; 1024^2: 31 %), and
// the warps wait for the busiest one at each step's barrier (10 cycles per
// issue) and for its gathers (7 to 9).  1.93 ms for 321 x 481, from 2.87 ms with
// bounds checks and a branch per neighbour.  Loading each level's place and
// columns a step ahead lengthened the busiest warp's step: 3.45 ms.
__global__ void __launch_bounds__(1024) k_ws_flood(const UcmImage* __restrict__ imgs, const int32_t* __restrict__ off,
                                                   const uint16_t* __restrict__ cols, int32_t* __restrict__ ws) {
  const UcmImage I = imgs[blockIdx.x];
  const int H = I.H, W = I.W, P = W + 2, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int32_t* L = ws + I.wpix + P + 1;  // pixel (0, 0)
  const int32_t* O = off + (long long)I.row0 * 257;
  const uint16_t* C = cols + I.pix;
  const int steps = 2 * 255 + H;
  for (int t = 0; t < steps; t++) {
    // this warp's levels whose row lies in the image
    const int lo = max(0, (t - H) / 2 + (t >= H)), hi = min(255, t / 2);
    for (int lvl = warp + ((max(lo - warp, 0) + 31) & ~31); lvl <= hi; lvl += 32) {
      const int x = t - 2 * lvl;
      const int b = O[x * 257 + lvl], e = O[x * 257 + lvl + 1];
      if (b >= e) continue;
      const uint16_t* row = C + (size_t)x * W;
      int32_t* Lr = L + (size_t)x * P;
      // column and the surrounding labels of the row's k-th pixel of the level
      // (past the last one: of the row's first pixel, unused)
      auto gather = [&](int k, int& y, int& left, int& mx, unsigned& mn) {
        const bool in = k < e;
        y = in ? (int)row[k] : -4;
        const int32_t* q = Lr + max(y, 0);
        const int v[7] = {q[-P - 1], q[-P], q[-P + 1], q[1], q[P - 1], q[P], q[P + 1]};
        left = q[-1];
        mx = v[0];
        mn = (unsigned)v[0] - 1u;  // labels > 0 as 0, 1, ..; 0 and -1 above all of them
#pragma unroll
        for (int i = 1; i < 7; i++) {
          mx = max(mx, v[i]);
          mn = min(mn, (unsigned)v[i] - 1u);
        }
      };
      int y, left, mx;
      unsigned mn;
      gather(b + lane, y, left, mx, mn);
      int carry = -1, ylast = -10;  // final label and column of the previous chunk's last pixel
      for (int k0 = b; k0 < e; k0 += 32) {
        const bool in = k0 + lane < e;
        int yn = -4, leftn = -1, mxn = -1;
        unsigned mnn = 0;
        if (k0 + 32 < e) gather(k0 + 32 + lane, yn, leftn, mxn, mnn);  // in flight while this chunk resolves
        const int yl = __shfl_up_sync(0xffffffffu, y, 1);
        const bool cross = in && lane == 0 && y - 1 == ylast;          // left pixel in the previous chunk
        const bool dep = in && (cross || (lane > 0 && yl == y - 1));  // left pixel is this level's, unresolved here
        if (!dep) {
          mx = max(mx, left);
          mn = min(mn, (unsigned)left - 1u);
        }
        // -1: no labelled neighbour, 0: two different labels, else the one label
        const int s = mx <= 0 ? -1 : ((int)mn + 1 == mx ? mx : 0);
        const int sl = __shfl_up_sync(0xffffffffu, s, 1);
        const int mine = x * W + y + 1;
        auto after = [&](int pv) {  // this pixel's label given the left pixel's
          return (s == -1) ? (pv > 0 ? pv : mine) : ((pv > 0 && pv != s) ? 0 : s);
        };
        int done, val;
        if (cross) {
          val = after(carry);
          done = 1;
        } else {
          // final without the left lane: no dependence, a conflict already, or
          // a label the left pixel can only repeat or have lost to a conflict
          done = !in || !dep || s == 0 || (s > 0 && (sl == s || sl == 0));
          val = !dep ? (s >= 0 ? s : mine) : s;
        }
        while (!__all_sync(0xffffffffu, done)) {
          const int pv = __shfl_up_sync(0xffffffffu, val, 1);
          const int pd = __shfl_up_sync(0xffffffffu, done, 1);
          if (!done && pd) {
            val = after(pv);
            done = 1;
          }
        }
        if (in) Lr[y] = val;
        if (k0 + 32 >= e) break;
        carry = __shfl_sync(0xffffffffu, val, 31);
        ylast = __shfl_sync(0xffffffffu, y, 31);
        __syncwarp();
        y = yn;
        left = leftn;
        mx = mxn;
        mn = mnn;
      }
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) k_ws_bw(UcmLaunch l, const int32_t* __restrict__ ws) {
  const UcmPart me = ucm_part(l);
  const UcmView& V = me.V;
  const int W = V.W, P = W + 2;
  const long long N = (long long)V.H * W;
  const int32_t* L = ws + V.s.img->wpix + P + 1;
  for (long long i = (long long)me.cta * blockDim.x + threadIdx.x; i < N; i += (long long)me.ctas * blockDim.x)
    V.s.bw[i] = L[i / W * P + i % W] == 0;
}

// ---------------------------------------------------------------- painting

// One thread per painted pixel: the edge's orientation plane at that pixel,
// max-ed into the strength map (which starts at 0, so negatives leave 0).
__global__ void __launch_bounds__(256) k_ucm_paint(UcmLaunch l) {
  const UcmPart me = ucm_part(l);
  const UcmView& V = me.V;
  const int32_t* __restrict__ pix = V.s.paint_pix;
  const uint8_t* __restrict__ ori = V.s.paint_ori;
  const int n = V.np;
  const long long N = (long long)V.H * V.W;
  const float* __restrict__ orient = V.orient;
  unsigned* wswt = (unsigned*)V.s.wswt;
  for (int i = me.cta * blockDim.x + threadIdx.x; i < n; i += me.ctas * blockDim.x) {
    const int p = pix[i];
    const float v = orient[(long long)ori[i] * N + p];
    if (v > 0.0f) atomicMax(wswt + p, __float_as_uint(v));  // non-negative floats order as their bits
  }
}

// ---------------------------------------------------------------- super contour

// pb2 (2H x 2W): even-even = ws_wt, even-odd = min of horizontal pairs,
// odd-even = min of vertical pairs, odd-odd = 0; the last row repeats the
// one before, the last column is max(itself, the one before).
__device__ __forceinline__ float super_base(const float* w, int H, int W, int r, int c) {
  const int i = r >> 1, j = c >> 1;
  if (!(r & 1) && !(c & 1)) return w[(size_t)i * W + j];
  if (!(r & 1) && (c & 1)) return c == 2 * W - 1 ? 0.0f : fminf(w[(size_t)i * W + j], w[(size_t)i * W + j + 1]);
  if ((r & 1) && !(c & 1)) return r == 2 * H - 1 ? 0.0f : fminf(w[(size_t)i * W + j], w[(size_t)(i + 1) * W + j]);
  return 0.0f;
}

__global__ void __launch_bounds__(256) k_ucm_super(UcmLaunch l) {
  const UcmPart me = ucm_part(l);
  const UcmView& V = me.V;
  const float* __restrict__ wswt = V.s.wswt;
  const int H = V.H, W = V.W;
  float* __restrict__ pb2 = V.s.pb2;
  const long long n = 4LL * H * W;
  const int W2 = 2 * W;
  for (long long k = (long long)me.cta * blockDim.x + threadIdx.x; k < n; k += (long long)me.ctas * blockDim.x) {
    int r = (int)(k / W2);
    const int c = (int)(k % W2);
    if (r == 2 * H - 1) r = 2 * H - 2;
    float v = super_base(wswt, H, W, r, c);
    if (c == W2 - 1) {
      const float a = v, b = super_base(wswt, H, W, r, c - 1);
      v = a < b ? b : a;
    }
    pb2[k] = v;
  }
}

// ---------------------------------------------------------------- artefacts

__device__ __forceinline__ bool isolated_zero(const float* g, int R, int C, int r, int c) {
  if (g[(size_t)r * C + c] != 0.0f) return false;
  for (int i = -1; i <= 1; i++)
    for (int j = -1; j <= 1; j++) {
      if (i == 0 && j == 0) continue;
      const int rr = r + i, cc = c + j;
      if (rr < 0 || rr >= R || cc < 0 || cc >= C) continue;
      if (g[(size_t)rr * C + cc] == 0.0f) return false;
    }
  return true;
}

// one warp per row: the row's isolated zeros, counted, or written in column
// order from the row's place (rowcnt, scanned)
template <bool WRITE>
__global__ void __launch_bounds__(32) k_art_rows(UcmLaunch l) {
  const UcmPart me = ucm_part<2>(l);
  const UcmView& V = me.V;
  const float* __restrict__ g = V.s.pb2;
  const int R = 2 * V.H, C = 2 * V.W;
  int32_t* __restrict__ list = V.s.art;
  const int r = me.cta, lane = threadIdx.x;
  if (r >= R) return;
  int k = WRITE ? V.s.rowcnt[r] : 0;
  for (int c0 = 0; c0 < C; c0 += 32) {
    const int c = c0 + lane;
    const bool hit = c < C && isolated_zero(g, R, C, r, c);
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (WRITE && hit) list[k + __popc(m & ((1u << lane) - 1u))] = r * C + c;
    k += __popc(m);
  }
  if (!WRITE && lane == 0) V.s.rowcnt[r] = k;
}

// exclusive scan in place by one CTA per image: of the rows' artefact counts
// (total to nart), or of the block sums of the root counts (total to nreg)
template <bool ROWS>
__global__ void __launch_bounds__(1024) k_scan_small(const UcmView* __restrict__ views) {
  const UcmView& V = views[blockIdx.x];
  int32_t* __restrict__ a = ROWS ? V.s.rowcnt : V.s.bsum;
  const int n = ROWS ? 2 * V.H : (int)((4LL * V.H * V.W + 4095) / 4096);
  int32_t* __restrict__ sum = ROWS ? V.s.nart : V.s.nreg;
  __shared__ int32_t part[1024];
  const int per = (n + 1023) / 1024, t = threadIdx.x, b = t * per;
  int32_t s = 0;
  for (int i = b; i < b + per && i < n; i++) s += a[i];
  part[t] = s;
  __syncthreads();
  for (int d = 1; d < 1024; d <<= 1) {
    const int32_t v = t >= d ? part[t - d] : 0;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  int32_t run = part[t] - s;
  for (int i = b; i < b + per && i < n; i++) {
    const int32_t v = a[i];
    a[i] = run;
    run += v;
  }
  if (t == 1023) *sum = part[1023];
}

// The fixes of CleanWatersheds in list order, one thread.  Reads outside
// the grid (artefacts within two cells of the border) read 0; writes there
// are dropped.
__global__ void k_art_fix(const UcmView* __restrict__ views) {
  const UcmView& V = views[blockIdx.x];
  float* __restrict__ g = V.s.pb2;
  const int R = 2 * V.H, C = 2 * V.W;
  const int32_t* __restrict__ list = V.s.art;
  const int32_t* __restrict__ n = V.s.nart;
  if (threadIdx.x) return;
  const long long tot = (long long)R * C;
  auto rd = [&](int r, int c) -> float {
    const long long k = (long long)r * C + c;  // a continuous matrix: columns wrap into the next row
    return (k >= 0 && k < tot) ? g[k] : 0.0f;
  };
  auto wr = [&](int r, int c, float v) {
    const long long k = (long long)r * C + c;
    if (k >= 0 && k < tot) g[k] = v;
  };
  for (int a = 0; a < *n; a++) {
    const int xc = list[a] / C, yc = list[a] % C;
    float vec[4];
    vec[0] = fmaxf(rd(xc - 2, yc - 1), rd(xc - 1, yc - 2));
    vec[1] = fmaxf(rd(xc + 2, yc - 1), rd(xc + 1, yc - 2));
    vec[2] = fmaxf(rd(xc + 2, yc + 1), rd(xc + 1, yc + 2));
    vec[3] = fmaxf(rd(xc - 2, yc + 1), rd(xc - 1, yc + 2));
    int id = 0;
    float nd = vec[0];
    for (int i = 1; i < 4; i++)
      if (vec[i] < nd) nd = vec[i], id = i;
    const int sx = (id == 1 || id == 2) ? 1 : -1, sy = (id >= 2) ? 1 : -1;
    const float p = rd(xc + 2 * sx, yc + sy), q = rd(xc + sx, yc + 2 * sy);
    if (p < q) {
      wr(xc, yc + sy, 0.0f);
      wr(xc + sx, yc, vec[id]);
    } else {
      wr(xc, yc + sy, vec[id]);
      wr(xc + sx, yc, 0.0f);
    }
    wr(xc + sx, yc + sy, vec[id]);
  }
}

// ---------------------------------------------------------------- labelling

__device__ __forceinline__ int ccl_find(const int32_t* p, int a) {
  int b = p[a];
  while (b != a) {
    a = b;
    b = p[a];
  }
  return a;
}

__device__ __forceinline__ void ccl_union(int32_t* p, int a, int b) {
  bool done = false;
  while (!done) {
    a = ccl_find(p, a);
    b = ccl_find(p, b);
    if (a == b) break;
    if (a < b) {
      const int t = a;
      a = b;
      b = t;
    }
    const int old = atomicMin(p + a, b);  // hang the larger root under the smaller
    done = (old == a);
    a = old;
  }
}

// one CTA per row, its warps taking segments of kCclSeg cells: every zero cell's
// parent is the first cell of its horizontal run in the segment, so the unions
// below only join runs of adjacent rows and segments.  (One warp per row took
// 834 us for rows of 120,000 cells, a thread per cell none of note; 222 us so.)
constexpr int kCclSeg = 512, kCclWarps = 4;
__global__ void __launch_bounds__(32 * kCclWarps) k_ccl_init(UcmLaunch l) {
  const UcmPart me = ucm_part<2>(l);
  const UcmView& V = me.V;
  const int R = 2 * V.H, C = 2 * V.W, r = me.cta, lane = threadIdx.x & 31;
  if (r >= R) return;
  const float* __restrict__ g = V.s.pb2 + (size_t)r * C;
  int32_t* __restrict__ p = V.s.par + (size_t)r * C;
  for (int s0 = (threadIdx.x >> 5) * kCclSeg; s0 < C; s0 += kCclWarps * kCclSeg) {
    int start = s0;  // the run that reaches the chunk's first cell begins here, if any does
    for (int c0 = s0; c0 < min(s0 + kCclSeg, C); c0 += 32) {
      const int c = c0 + lane;
      const bool zero = c < C && __ldg(g + c) == 0.0f;
      const unsigned walls = ~__ballot_sync(0xffffffffu, zero);
      const unsigned before = walls & ((1u << lane) - 1u);
      if (c < C) p[c] = zero ? r * C + (before ? c0 + 32 - __clz(before) : start) : -1;
      if (walls) start = c0 + 32 - __clz(walls);
    }
  }
}

// Joins with the row above, one union per contact of two runs (12 us for a
// 642 x 962 grid, from 163 us with a union per adjacent pair): with the cell
// above unless the left neighbour already has that contact; with a diagonal
// cell only where the cells between offer none; and with the left cell where a
// segment begins.
__global__ void __launch_bounds__(256) k_ccl_hook(UcmLaunch l) {
  const UcmPart me = ucm_part(l);
  const UcmView& V = me.V;
  const float* __restrict__ g = V.s.pb2;
  int32_t* p = V.s.par;
  const int R = 2 * V.H, C = 2 * V.W;
  const long long n = (long long)R * C;
  for (long long k = (long long)me.cta * blockDim.x + threadIdx.x; k < n; k += (long long)me.ctas * blockDim.x) {
    if (g[k] != 0.0f) continue;
    const int c = (int)(k % C);
    const bool left = c > 0 && g[k - 1] == 0.0f;
    if (left && c % kCclSeg == 0) ccl_union(p, (int)k, (int)k - 1);
    if (k < C) continue;
    const bool upleft = c > 0 && g[k - C - 1] == 0.0f;
    if (g[k - C] == 0.0f) {
      if (!(left && upleft)) ccl_union(p, (int)k, (int)(k - C));
      continue;
    }
    if (upleft && !left) ccl_union(p, (int)k, (int)(k - C - 1));
    if (c + 1 < C && g[k - C + 1] == 0.0f && g[k + 1] != 0.0f) ccl_union(p, (int)k, (int)(k - C + 1));
  }
}

// flatten to roots; rank[k] = 1 where k is a root (the component's first cell)
__global__ void __launch_bounds__(256) k_ccl_flat(UcmLaunch l) {
  const UcmPart me = ucm_part(l);
  const UcmView& V = me.V;
  int32_t* p = V.s.par;
  int32_t* __restrict__ root = V.s.rank;
  const long long n = 4LL * V.H * V.W;
  for (long long k = (long long)me.cta * blockDim.x + threadIdx.x; k < n; k += (long long)me.ctas * blockDim.x) {
    if (p[k] < 0) {
      root[k] = 0;
      continue;
    }
    const int r = ccl_find(p, (int)k);
    p[k] = r;
    root[k] = r == k;
  }
}

// region labels of the pixels (0-based; cells that are not zeros give -1)
// and ws_wt2, the grid padded by its last row and column
__global__ void __launch_bounds__(256) k_ucm_finish(UcmLaunch l) {
  const UcmPart me = ucm_part(l);
  const UcmView& V = me.V;
  const float* __restrict__ g = V.s.pb2;
  const int32_t* __restrict__ p = V.s.par;
  const int32_t* __restrict__ rank = V.s.rank;
  const int H = V.H, W = V.W;
  int32_t* __restrict__ labels = V.s.labels;
  float* __restrict__ wswt2 = V.s.wswt2;
  const int R = 2 * H, C = 2 * W;
  const long long n2 = (long long)(R + 1) * (C + 1);
  for (long long k = (long long)me.cta * blockDim.x + threadIdx.x; k < n2; k += (long long)me.ctas * blockDim.x) {
    const int r = (int)(k / (C + 1)), c = (int)(k % (C + 1));
    wswt2[k] = g[(size_t)(r == R ? R - 1 : r) * C + (c == C ? C - 1 : c)];
    if (r < H && c < W) {
      const long long cell = (long long)(2 * r + 1) * C + 2 * c + 1;
      const int32_t root = p[cell];
      labels[(size_t)r * W + c] = root < 0 ? -1 : rank[root];  // rank is the exclusive count of roots before
    }
  }
}

// exclusive scan of n (up to 2^31) ints through blocks of 1024 x 4
__global__ void __launch_bounds__(1024) k_scan_blocks(UcmLaunch l) {
  const UcmPart me = ucm_part(l);
  const UcmView& V = me.V;
  int32_t* __restrict__ a = V.s.rank;
  int32_t* __restrict__ bsum = V.s.bsum;
  const long long n = 4LL * V.H * V.W;
  if ((long long)me.cta * 4096 >= n) return;
  __shared__ int32_t part[1024];
  const long long b0 = (long long)me.cta * 4096;
  const int t = threadIdx.x;
  int32_t v[4], s = 0;
  for (int k = 0; k < 4; k++) {
    const long long i = b0 + t * 4 + k;
    v[k] = i < n ? a[i] : 0;
    s += v[k];
  }
  part[t] = s;
  __syncthreads();
  for (int d = 1; d < 1024; d <<= 1) {
    const int32_t u = t >= d ? part[t - d] : 0;
    __syncthreads();
    part[t] += u;
    __syncthreads();
  }
  int32_t run = part[t] - s;
  for (int k = 0; k < 4; k++) {
    const long long i = b0 + t * 4 + k;
    if (i < n) a[i] = run;
    run += v[k];
  }
  if (t == 1023) bsum[me.cta] = part[1023];
}

__global__ void __launch_bounds__(256) k_scan_add(UcmLaunch l) {
  const UcmPart me = ucm_part(l);
  const UcmView& V = me.V;
  int32_t* __restrict__ a = V.s.rank;
  const int32_t* __restrict__ bsum = V.s.bsum;
  const long long n = 4LL * V.H * V.W;
  for (long long i = (long long)me.cta * blockDim.x + threadIdx.x; i < n; i += (long long)me.ctas * blockDim.x)
    a[i] += bsum[i / 4096];
}

// ---------------------------------------------------------------- launchers

static int grid_for(long long n) {
  const long long g = (n + 255) / 256;
  return (int)(g < 1 ? 1 : (g > 152 * 16 ? 152 * 16 : g));
}

void ucm_ctas(UcmView* views, UcmBatch& b) {
  int at[kUcmKinds] = {};
  for (int i = 0; i <= b.n; i++) {
    std::copy(at, at + kUcmKinds, views[i].first);
    if (i == b.n) break;
    const long long N = (long long)views[i].H * views[i].W;
    at[kUcmPix] += grid_for(N);
    at[kUcmCells] += grid_for(4 * N);
    at[kUcmRows] += views[i].H;
    at[kUcmPaint] += views[i].np ? grid_for(views[i].np) : 0;
    at[kUcmScan] += (int)((4 * N + 4095) / 4096);
  }
  std::copy(at, at + kUcmKinds, b.ctas);
}

static UcmLaunch ucm_launch(const UcmBatch& b, UcmKind k) { return {b.views, b.n, k}; }

cudaError_t ucm_prepare(const UcmBatch& b, const UcmScratch& base, cudaStream_t st) {
  const cudaError_t e = cudaMemsetAsync(base.mm, 0, 2 * (size_t)b.n * sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  k_ucm_pbmax<<<b.ctas[kUcmPix], 256, 0, st>>>(ucm_launch(b, kUcmPix));
  k_ucm_quant<<<b.ctas[kUcmPix], 256, 0, st>>>(ucm_launch(b, kUcmPix));
  k_ws_rowsort<<<b.ctas[kUcmRows], 32, 0, st>>>(ucm_launch(b, kUcmRows));
  return cudaGetLastError();
}

cudaError_t ucm_flood(const UcmBatch& b, const UcmScratch& base, cudaStream_t st) {
  const cudaError_t e = cudaMemsetAsync(base.ws, 0xff, (size_t)b.ws_cells * sizeof(int32_t), st);
  if (e != cudaSuccess) return e;
  k_ws_flood<<<b.n, 1024, 0, st>>>(base.img, base.off, base.cols, base.ws);
  k_ws_bw<<<b.ctas[kUcmPix], 256, 0, st>>>(ucm_launch(b, kUcmPix), base.ws);
  return cudaGetLastError();
}

cudaError_t ucm_paint(const UcmBatch& b, const UcmScratch& base, cudaStream_t st) {
  const cudaError_t e = cudaMemsetAsync(base.wswt, 0, (size_t)b.total_pix * sizeof(float), st);
  if (e != cudaSuccess) return e;
  if (b.ctas[kUcmPaint] > 0) k_ucm_paint<<<b.ctas[kUcmPaint], 256, 0, st>>>(ucm_launch(b, kUcmPaint));
  return cudaGetLastError();
}

cudaError_t ucm_mid(const UcmBatch& b, cudaStream_t st) {
  const UcmLaunch cells = ucm_launch(b, kUcmCells), rows = ucm_launch(b, kUcmRows);
  const int nc = b.ctas[kUcmCells], nr = 2 * b.ctas[kUcmRows];  // rows of the doubled grid
  k_ucm_super<<<nc, 256, 0, st>>>(cells);
  k_art_rows<false><<<nr, 32, 0, st>>>(rows);
  k_scan_small<true><<<b.n, 1024, 0, st>>>(b.views);
  k_art_rows<true><<<nr, 32, 0, st>>>(rows);
  k_art_fix<<<b.n, 32, 0, st>>>(b.views);
  k_ccl_init<<<nr, 32 * kCclWarps, 0, st>>>(rows);
  k_ccl_hook<<<nc, 256, 0, st>>>(cells);
  k_ccl_flat<<<nc, 256, 0, st>>>(cells);
  k_scan_blocks<<<b.ctas[kUcmScan], 1024, 0, st>>>(ucm_launch(b, kUcmScan));
  k_scan_small<false><<<b.n, 1024, 0, st>>>(b.views);
  k_scan_add<<<nc, 256, 0, st>>>(cells);
  k_ucm_finish<<<nc, 256, 0, st>>>(cells);
  return cudaGetLastError();
}

}  // namespace gpb
