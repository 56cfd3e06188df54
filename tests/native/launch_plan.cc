// The launch rules of csrc/gpu/plan.h over every SM count up to 200 (a partition of the part
// reports fewer than the whole) and every size: what a launch writes has to fit its buffer.
#include "../../flock_gb300/csrc/gpu/plan.h"
#include <cstdio>

using namespace flock::gpu;

static int failures = 0;
static void expect(bool ok, const char* what, uint64_t a, uint64_t b) {
  if (ok) return;
  if (++failures <= 10) printf("%s: %llu, %llu\n", what, (unsigned long long)a, (unsigned long long)b);
}

// The assist's launches over n dense words: the build, then a fold a round.
static void assist_partials_fit() {
  for (uint64_t sms = 1; sms <= 200; ++sms)
    for (uint32_t m = 5; m <= 28; ++m) {
      const uint64_t n = uint64_t(1) << m, room = assist_partials(n, sms);
      expect(2 * as_build_blocks(n, sms) <= room, "assist build: SMs, m", sms, m);
      for (uint64_t len = n; len >= 4; len /= 2)
        expect(2 * pair_fold_plan(len / 4, EQ_NONE, 0, false, sms).blocks <= room, "assist fold: SMs, length", sms, len);
    }
}

int main() {
  assist_partials_fit();
  printf("failures %d\n", failures);
  return failures != 0;
}
