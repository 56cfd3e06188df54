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

// The weighted zerocheck's division (round w) is a device round: the fold that leaves the host's
// tail of 2^TAIL_LOG entries, round L - TAIL_LOG, or one before it.
static void division_before_the_tail() {
  for (uint64_t sms = 1; sms <= 200; ++sms)
    for (uint32_t L = 10; L <= 28; ++L)
      for (uint64_t live = uint64_t(1) << (L - 1); live <= uint64_t(1) << L; live += uint64_t(1) << (L - 5)) {
        const uint32_t w = zc_weighted_lo_bits(live, L, sms);
        expect(w == 0 || (w >= 10 && w <= 12 && w + TAIL_LOG <= L), "weighted rounds: SMs, L", sms, L);
      }
  // the whole part's choices: BLAKE3 2^10 and 2^11, Keccak-f 2^9, SHA-256 2^13, Keccak-f 2^13
  expect(zc_weighted_lo_bits(92 << 10, 17, 152) == 0, "plain", 17, 152);
  expect(zc_weighted_lo_bits(92 << 11, 18, 152) == 10, "chunks of 2^10", 18, 152);
  expect(zc_weighted_lo_bits(333 << 9, 18, 152) == 10, "chunks of 2^10", 18, 152);
  expect(zc_weighted_lo_bits(199 << 13, 21, 152) == 11, "chunks of 2^11", 21, 152);
  expect(zc_weighted_lo_bits(333 << 13, 22, 152) == 12, "chunks of 2^12", 22, 152);
}

// The bit sums' partials: round 1 (64 columns, half of the buffer for 128 a row), the lane dots (up to
// 64 lanes), the lincheck's row fold (as many splits as the buffer has room for).
static void bit_sums_fit() {
  for (uint64_t sms = 1; sms <= 200; ++sms)
    for (uint32_t k = 0; k <= 26; ++k)
      for (uint64_t rows : {uint64_t(1) << k, (uint64_t(1) << k) + (uint64_t(1) << k / 2) + 1}) {
        const BitSumPlan r1 = bit_sum_plan(64, rows, BITS_MAX_SPLITS, sms);
        expect(uint64_t(r1.groups) * r1.splits * 128 <= PART_ENTRIES / 2, "round 1: SMs, rows", sms, rows);
        for (uint32_t cols : {1u, 13u, 42u, 64u, 333u, 1024u}) {
          const bool wide = cols > 64;
          const BitSumPlan p = bit_sum_plan(cols, rows, wide ? PART_ENTRIES / (cols * 128ull) : BITS_MAX_SPLITS, sms);
          expect(uint64_t(p.splits) * cols * (wide ? 128 : 1) <= PART_ENTRIES, "bit sums: SMs, rows", sms, rows);
          expect(p.splits * p.rows_per_split >= rows && uint64_t(p.groups) * p.cpw * BITS_WARPS >= cols, "cover: SMs, rows", sms, rows);
        }
      }
}

int main() {
  bit_sums_fit();
  division_before_the_tail();
  assist_partials_fit();
  fold_partials_fit();
  printf("failures %d\n", failures);
  return failures != 0;
}
