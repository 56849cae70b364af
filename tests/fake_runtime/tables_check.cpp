// Disc offsets that do not fit the cue kernel's table: an error, not an abort.
#include "fake_runtime.h"

#include <stdio.h>

#include "gpb_internal.h"
#include "kernels.h"

using namespace gpb;

int main() {
  HostTables t;
  build_tables(t, 0);
  if (upload_cues(t, nullptr) != cudaSuccess) return printf("the tables were refused\n"), 1;
  t.ann_count[0][0] += 100;
  if (upload_cues(t, nullptr) == cudaSuccess) return printf("taken\n"), 1;
  printf("ok\n");
  return 0;
}
