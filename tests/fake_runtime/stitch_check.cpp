// CTAs of a stitch: in proportion to the boxes (32 x 32 pixels each), however
// large the image and however far apart the boxes, and none for boxes outside.
#include "fake_runtime.h"

#include <stdio.h>

#include "kernels.h"

using namespace gpb;

static int bad = 0;
static double ctas(std::vector<StitchBox> b, int w, int h, bool blend) {
  fake().launches.clear();
  std::vector<StitchSpan> dev(b.size());
  const cudaError_t e = launch_stitch(nullptr, b.data(), b.size() > (size_t)kStitchFew ? dev.data() : nullptr,
                                      (int)b.size(), blend, nullptr, nullptr, 0, w, h, 4.f, nullptr, nullptr, nullptr);
  if (e != cudaSuccess) bad++;
  return fake().ctas("k_stitch");
}
#define AT_MOST(n, c)                                                \
  do {                                                               \
    const double v = (c);                                            \
    if (v > (n)) printf("line %d: %.0f > %.0f\n", __LINE__, v, (double)(n)), bad++; \
  } while (0)

int main() {
  for (int blend = 0; blend < 2; blend++) {
    AT_MOST(81, ctas({{40, 40, 0, 0, 256, 256}}, 16384, 16384, blend));
    AT_MOST(2 * 81, ctas({{0, 0, 0, 0, 256, 256}, {16100, 16000, 0, 0, 256, 256}}, 16384, 16384, blend));
    std::vector<StitchBox> grid, scattered;
    for (int i = 0; i < 16; i++) grid.push_back({256 * (i % 4) - 5, 256 * (i / 4) - 5, 0, 0, 266, 266});
    AT_MOST(1024, ctas(grid, 1024, 1024, blend));
    for (int i = 0; i < 200; i++) scattered.push_back({(i * 7919) % 8000, (i * 104729) % 8000, 0, 0, 33, 40});
    AT_MOST(200 * 9, ctas(scattered, 8192, 8192, blend));
    AT_MOST(0, ctas({{-300, 5, 0, 0, 256, 256}, {900, 1024, 0, 0, 64, 64}, {3, 3, 5, 5, 0, 7}}, 1024, 1024, blend));
    AT_MOST(4, ctas({{0x7fffffff - 32, 0, 0, 0, 64, 32}}, 0x7fffffff, 33, blend));
  }
  if (!bad) printf("ok\n");
  return bad != 0;
}
