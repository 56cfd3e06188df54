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

// Every fold's partials, the plain form's on large vectors among them.
static void fold_partials_fit() {
  for (uint64_t sms = 1; sms <= 200; ++sms)
    for (uint64_t pairs = 1; pairs <= uint64_t(1) << 30; pairs *= 2)
      for (PairEq eq : {EQ_NONE, EQ_FIXED, EQ_SPLIT})
        for (uint32_t lo = 0; lo <= 11; ++lo)
          for (bool unweight : {false, true}) {
            const PairFoldPlan p = pair_fold_plan(pairs, eq, lo, unweight, sms);
            expect(p.blocks >= 1 && 2 * uint64_t(p.blocks) <= PART_ENTRIES, "fold partials: SMs, pairs", sms, pairs);
          }
}

int main() {
  assist_partials_fit();
  fold_partials_fit();
  printf("failures %d\n", failures);
  return failures != 0;
}
