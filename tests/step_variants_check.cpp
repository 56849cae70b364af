// cf_launch_step's variants on the GPU: the fine and the coarse stencil, plain
// and compensated, with and without the third term, over patches whose last
// 16 x 16 tiles are cut at 1, 8, 9 and 16 rows.  Both variants equal to the bit,
// and within the rounding bound of the sums in FP64.
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <vector>

#include "k_block.h"

using namespace gpb;

static unsigned long long seed = 88172645463325252ull;
static float rnd() {
  seed ^= seed << 13, seed ^= seed >> 7, seed ^= seed << 17;
  return (float)(seed >> 40) / 8388608.f - 1.f;
}
template <class T>
static T* up(const std::vector<T>& v) {
  T* p = nullptr;
  if (cudaMalloc(&p, v.size() * sizeof(T)) != cudaSuccess) return nullptr;
  cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
  return p;
}

static int check(bool coarse) {
  const int sizes[][2] = {{33, 47}, {40, 64}, {41, 35}, {48, 32}, {32, 49}, {17, 200}, {64, 33}};
  const int R = coarse ? 3 : 5, nc = coarse ? kCoarseNC : kFullNC, np = 7;
  std::vector<int> dy, dx;
  for (int y = -R; y <= R; y++)
    for (int x = -R; x <= R; x++)
      if (coarse || y * y + x * x <= 25) dy.push_back(y), dx.push_back(x);
  std::vector<PatchDev> patches(np);
  std::vector<int4> work;
  const long long pad = 5 * 200 + 5 + 16 + 10 + 64;
  long long vec = pad;
  for (int i = 0; i < np; i++) {
    PatchDev& P = patches[i];
    memset(&P, 0, sizeof(P));
    P.H = sizes[i][0], P.W = sizes[i][1], P.N = P.H * P.W, P.vec = vec;
    vec += P.N + pad;
    for (int y = 0; y < P.H; y += 16)
      for (int x = 0; x < P.W; x += 16) work.push_back(make_int4(i, y, x, (int)work.size()));
  }
  std::vector<float> Y(vec * kBlk), X(vec * kBlk), A((size_t)work.size() * 256 * nc);
  std::vector<int> active(np, 1), err(1, 0);
  active[3] = 0;
  const int steps = 2;
  std::vector<float3> coef(np * steps);
  for (int i = 0; i < np; i++) {
    coef[i * steps] = make_float3(1.f + rnd(), rnd(), 0.f);
    coef[i * steps + 1] = make_float3(1.f + rnd(), rnd(), rnd());
    for (long long q = patches[i].vec * kBlk; q < (patches[i].vec + patches[i].N) * kBlk; q++) Y[q] = rnd(), X[q] = rnd();
  }
  auto at = [&](size_t tile, int slot, int e) { return ((tile * (nc / 4) + e / 4) * 256 + slot) * 4 + e % 4; };
  for (const int4& t : work) {
    const PatchDev& P = patches[t.x];
    for (int s = 0; s < 256; s++) {
      const int k = (s >> 2) & 7, y = t.y + 2 * (s >> 5) + (k >> 2), x = t.z + 4 * (s & 3) + (k & 3);
      for (size_t e = 0; e < dy.size(); e++) {
        const int yy = y + dy[e], xx = x + dx[e];
        if (y < P.H && x < P.W && yy >= 0 && yy < P.H && xx >= 0 && xx < P.W) A[at(t.w, s, (int)e)] = rnd();
      }
    }
  }
  BlkArgs a = {};
  a.patches = up(patches), a.active = up(active), a.coef = up(coef), a.max_steps = steps;
  a.afull = up(A), a.err = up(err), a.coarse = coarse;
  const int4* w = up(work);
  const float *dY = up(Y), *dX = up(X);
  std::vector<float> blank(Y.size(), -7.f);
  float* out = up(blank);
  if (!out) return printf("no memory\n"), 1;
  for (int comp = 0; comp < 2; comp++)
    for (int step = 0; step < steps; step++) {
      std::vector<float> got[kStepVariants];
      for (int v = 0; v < kStepVariants; v++) {
        cudaMemcpy(out, blank.data(), blank.size() * 4, cudaMemcpyHostToDevice);
        if (cf_launch_step(a, w, (int)work.size(), dY, dX, out, step, 0, comp, v) != cudaSuccess ||
            cudaDeviceSynchronize() != cudaSuccess)
          return printf("launch failed\n"), 1;
        got[v].resize(blank.size());
        cudaMemcpy(got[v].data(), out, blank.size() * 4, cudaMemcpyDeviceToHost);
        if (memcmp(got[v].data(), got[0].data(), blank.size() * 4))
          return printf("coarse %d comp %d step %d: variant %d differs\n", coarse, comp, step, v), 1;
      }
      cudaMemcpy(err.data(), a.err, 4, cudaMemcpyDeviceToHost);
      if (err[0]) return printf("a wait gave up\n"), 1;
      std::vector<char> seen(blank.size(), 0);
      for (const int4& t : work) {
        if (!active[t.x]) continue;
        const PatchDev& P = patches[t.x];
        const float3 c = coef[t.x * steps + step];
        for (int s = 0; s < 256; s++) {
          const int k = (s >> 2) & 7, y = t.y + 2 * (s >> 5) + (k >> 2), x = t.z + 4 * (s & 3) + (k & 3);
          if (y >= P.H || x >= P.W) continue;
          const long long q = P.vec + (long long)y * P.W + x;
          for (int j = 0; j < kBlk; j++) {
            double sum = 0, mag = 0;
            for (size_t e = 0; e < dy.size(); e++) {
              const float f = A[at(t.w, s, (int)e)];
              if (f == 0) continue;
              const double m = (double)f * Y[(q + (long long)dy[e] * P.W + dx[e]) * kBlk + j];
              sum += m, mag += fabs(m);
            }
            const double ty = (double)c.y * Y[q * kBlk + j], tx = (double)c.z * X[q * kBlk + j];
            const double want = c.x * sum + ty + tx, bound = 84 * ldexp(1, -24) * (fabs(c.x) * mag + fabs(ty) + fabs(tx));
            if (!(fabs(got[0][q * kBlk + j] - want) <= bound))
              return printf("coarse %d comp %d step %d patch %d (%d, %d): %g for %g\n", coarse, comp, step, t.x, y, x,
                            got[0][q * kBlk + j], want), 1;
            seen[q * kBlk + j] = 1;
          }
        }
      }
      for (size_t i = 0; i < blank.size(); i++)
        if (!seen[i] && got[0][i] != -7.f) return printf("wrote outside the active patches\n"), 1;
    }
  return 0;
}

int main() {
  if (check(false) || check(true)) return 1;
  printf("ok\n");
  return 0;
}
