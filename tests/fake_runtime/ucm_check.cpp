// A batch of one long image and thousands of tiny ones: the CTAs of every
// launch are in proportion to the images' own rows and pixels.
#include "fake_runtime.h"

#include <stdio.h>

#include "gpb.h"

int main() {
  const size_t n = 6001;
  std::vector<uint32_t> w(n, 2), h(n, 2);
  h[n / 2] = 6000;
  std::vector<float> planes(8 * 6000 * 2);
  std::vector<const float*> in(n, planes.data());
  std::vector<double> out(12001 * 5);
  std::vector<double*> outs(n, out.data());
  gpb_ctx* ctx = nullptr;
  if (gpb_create(&ctx, nullptr) != GPB_OK) return printf("no context\n"), 1;
  fake().launches.clear();
  const gpb_status st = gpb_ucm_batch(ctx, n, w.data(), h.data(), in.data(), 0, 1, outs.data(), nullptr);
  if (st != GPB_OK) return printf("status %d\n", (int)st), 1;
  double most = 0;
  for (size_t i = 0; i < n; i++) most += 2 * h[i] + 4 * w[i] * h[i] / 256 + 1;
  int bad = 0;
  for (const FakeLaunch& l : fake().launches) {
    const double c = (double)l.grid.x * l.grid.y * l.grid.z;
    if (c > most) printf("%s: %.0f CTAs, %.0f at most\n", l.kernel.c_str(), c, most), bad++;
  }
  if (fake().launches.size() < 12) printf("%zu launches\n", fake().launches.size()), bad++;
  gpb_destroy(ctx);
  if (!bad) printf("ok\n");
  return bad != 0;
}
