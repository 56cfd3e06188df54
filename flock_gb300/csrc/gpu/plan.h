// Launch shapes and buffer sizes that follow from a size and the SM count. No CUDA in here, so
// that a host test can walk every SM count (a partition of the part reports fewer than 152).
#pragma once
#include <algorithm>
#include <cstdint>

namespace flock {
namespace gpu {

constexpr uint32_t PART_ENTRIES = 1u << 20;  // a backend's buffer of per-block partials

// ------------------------------------------------------------------ bit sums
constexpr uint32_t BITS_THREADS = 512, BITS_WARPS = BITS_THREADS / 32;
constexpr uint32_t BITS_MAX_SPLITS = 1024;  // partial rows of round 1 and of the lane dots
// Columns per warp and row splits: the pair of least time, for blocks that cost about 105 cycles a
// tile and column slot (used or not), 700 for the tile's tables and 6000 + 4000 a column slot of
// the warp for its start and end (the latter is what counts where there are few rows), one block
// per SM at a time; at most max_splits partial rows and at least a tile each.
struct BitSumPlan {
  uint32_t cpw, groups, splits;
  uint64_t rows_per_split;
};
inline BitSumPlan bit_sum_plan(uint32_t n_cols, uint64_t n_rows, uint64_t max_splits, uint64_t sms) {
  BitSumPlan p{};
  const uint64_t tiles = (n_rows + 31) / 32;
  max_splits = std::max<uint64_t>(1, std::min(max_splits, tiles));
  uint64_t best = ~0ull;
  for (uint32_t cpw = 1; cpw <= 4; ++cpw) {
    const uint32_t groups = (n_cols + BITS_WARPS * cpw - 1) / (BITS_WARPS * cpw);
    for (uint64_t waves = 1; waves <= 4; ++waves) {
      const uint64_t want = std::min(max_splits, std::max<uint64_t>(1, waves * sms / groups));
      const uint64_t per = (tiles + want - 1) / want, splits = (tiles + per - 1) / per;
      const uint64_t used = (splits * groups + sms - 1) / sms;
      const uint64_t cost = used * (per * (105 * BITS_WARPS * cpw + 700) + 4000 * cpw + 6000);
      if (cost < best) {
        best = cost;
        p = {cpw, groups, (uint32_t)splits, per * 32};
      }
    }
  }
  return p;
}

// ------------------------------------------------------------------ pair folds
// Folds of at least this many pairs take the table form (see the kernels in sumcheck.cu).
constexpr uint64_t PAIR_FOLD_TABLE_MIN_PAIRS = uint64_t(1) << 17;
constexpr uint32_t PAIR_FOLD_TABLE_THREADS = 512;
constexpr uint32_t SMALL_PAIRS = 64;  // of a block of the small form
enum PairEq : int {
  EQ_NONE,   // eq = 1
  EQ_FIXED,  // eq(j) = eq_lo[j mod 2^lo_bits] (the zerocheck's weighted form); in the table form the
             // grid's thread count is a multiple of 2^lo_bits, so a thread multiplies its sum once
  EQ_SPLIT,  // eq(j) = eq_lo[j mod 2^lo_bits] eq_hi[j >> lo_bits]
};
struct PairFoldPlan {
  bool table;
  uint32_t blocks;  // each writes two partials
};
// The small form's widest grid: what its folds below the table form take. Larger ones (the
// zerocheck's plain form on a large vector, after a challenge the weighted form cannot divide by)
// walk their pairs with it, so that their partials have room at any size.
constexpr uint32_t PAIR_FOLD_SMALL_BLOCKS = PAIR_FOLD_TABLE_MIN_PAIRS / SMALL_PAIRS;
inline PairFoldPlan pair_fold_plan(uint64_t n_pairs, PairEq eq, uint32_t lo_bits, bool unweight, uint64_t sms) {
  if (n_pairs < PAIR_FOLD_TABLE_MIN_PAIRS || eq == EQ_SPLIT || unweight)
    return {false, (uint32_t)std::min<uint64_t>((n_pairs + SMALL_PAIRS - 1) / SMALL_PAIRS, PAIR_FOLD_SMALL_BLOCKS)};
  // one block per SM; under EQ_FIXED a multiple of 2^lo_bits threads in all
  uint32_t blocks = (uint32_t)sms;
  if (eq == EQ_FIXED && (1u << lo_bits) > PAIR_FOLD_TABLE_THREADS) {
    const uint32_t q = (1u << lo_bits) / PAIR_FOLD_TABLE_THREADS;
    blocks = std::max(q, blocks / q * q);
  }
  return {true, blocks};
}

// ------------------------------------------------------------------ zerocheck, weighted form
// Entries that a sumcheck's last device fold leaves for the host (GpuBackend::TailPair).
constexpr uint32_t TAIL_LOG = 7;
// Low bits of the chunks of the weighted form over 2^L words, `live_words` of them live; 0 where
// the plain form runs. A chunk's tables are rebuilt for it (about 2000 cycles beside 13 a word), so
// chunks are as long as leaves every SM four, down to 2^10 words with one an SM; smaller vectors
// take the plain form, whose launches are bound by latency. Round w of 2^w-word chunks divides by
// the chunks' weights, and has to be a device round: round L - TAIL_LOG is the last one.
inline uint32_t zc_weighted_lo_bits(uint64_t live_words, uint32_t L, uint64_t sms) {
  if ((live_words >> 12) >= 4 * sms && 12 + TAIL_LOG <= L) return 12;
  if ((live_words >> 11) >= 4 * sms && 11 + TAIL_LOG <= L) return 11;
  return (live_words >> 10) >= sms && 10 + TAIL_LOG <= L ? 10 : 0;
}

// ------------------------------------------------------------------ the jagged assist
constexpr uint32_t AS_BUILD_THREADS = 512;
inline uint32_t as_build_blocks(uint64_t n, uint64_t sms) {
  return (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((n / 2 + AS_BUILD_THREADS - 1) / AS_BUILD_THREADS, sms));
}
// Partials that the assist over n dense words needs room for: two a block of its widest launch
// (the first small fold has 1024 blocks, whatever the SM count).
inline uint64_t assist_partials(uint64_t n, uint64_t sms) {
  uint64_t blocks = as_build_blocks(n, sms);
  for (uint64_t pairs = n / 4; pairs; pairs /= 2)
    blocks = std::max<uint64_t>(blocks, pair_fold_plan(pairs, EQ_NONE, 0, false, sms).blocks);
  return 2 * blocks;
}

}  // namespace gpu
}  // namespace flock
