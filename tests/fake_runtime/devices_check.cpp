// Contexts on two devices, used by two threads each from the first call on:
// every launch must find its kernel's shared memory already granted on its own
// device, and a refusal to grant it must reach the caller.
#include "fake_runtime.h"

#include <stdio.h>

#include "gpb.h"
#include "k_block.h"
#include "kernels.h"

using namespace gpb;

static std::mutex bad_mu;
static int bad = 0;
#define CHECK(c)                                          \
  do {                                                    \
    if (!(c)) {                                           \
      std::lock_guard<std::mutex> lk(bad_mu);             \
      printf("check failed line %d: %s\n", __LINE__, #c); \
      bad++;                                              \
    }                                                     \
  } while (0)

static cudaError_t every_launch() {
  cudaError_t first = cudaSuccess;
  auto keep = [&](cudaError_t e) {
    if (first == cudaSuccess) first = e;
  };
  BlkArgs a = {};
  for (int coarse = 0; coarse < 2; coarse++)
    for (int comp = 0; comp < 2; comp++)
      for (int v = 0; v < kStepVariants; v++) {
        a.coarse = coarse;
        keep(cf_launch_step(a, nullptr, 40, nullptr, nullptr, nullptr, 0, nullptr, comp, v));
      }
  double g[1];
  keep(cf_launch_gram(a, 1, 3, nullptr, nullptr, g, nullptr));
  keep(cf_launch_gram(a, 1, 3, nullptr, nullptr, g, nullptr, g));
  keep(cf_launch_rotate(a, 3, nullptr, nullptr, kBlk, nullptr, false));
  keep(cf_launch_rotate(a, 3, nullptr, nullptr, kBlk, nullptr, true));
  float raw[1];
  keep(launch_cues(nullptr, nullptr, 4, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr));
  keep(launch_cues(nullptr, nullptr, 4, nullptr, nullptr, nullptr, nullptr, raw, nullptr, nullptr));
  return first;
}

// the network's convolutions and weight gradients, all layers
static gpb_status gradient(int device) {
  gpb_params p;
  gpb_default_params(&p);
  p.device = device;
  gpb_ctx* ctx = nullptr;
  gpb_status st = gpb_create(&ctx, &p);
  if (st != GPB_OK) return st;
  const size_t np = gpb_learned_nparams();
  std::vector<float> w(np, 0.f), g(np), x(16 * 16 * 9);
  const uint32_t side = 16;
  double loss = 0;
  st = gpb_learned_set(ctx, w.data(), np);
  if (st == GPB_OK) st = gpb_learned_grad_device(ctx, 1, &side, &side, x.data(), x.data(), x.data(), &loss, g.data());
  gpb_destroy(ctx);
  return st;
}

int main(int argc, char** argv) {
  if (argc > 1) {  // grants fail at first
    fake().fail_attributes = true;
    CHECK(every_launch() != cudaSuccess);
    CHECK(gradient(0) != GPB_OK);
    CHECK(fake().refused == 0);  // nothing is launched without its grant
    fake().fail_attributes = false;
  }
  std::vector<std::thread> t;
  for (int i = 0; i < 4; i++)
    t.emplace_back([i] {
      cudaSetDevice(i & 1);
      CHECK(every_launch() == cudaSuccess);
      CHECK(gradient(i & 1) == GPB_OK);
    });
  for (auto& x : t) x.join();
  CHECK(fake().refused == 0);
  for (int d = 0; d < 2; d++) {
    int n = 0;
    for (const FakeLaunch& l : fake().launches) n += l.device == d && l.smem > 48 * 1024;
    CHECK(n > 0);
  }
  if (!bad) printf("ok\n");
  return bad != 0;
}
