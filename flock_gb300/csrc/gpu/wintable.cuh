// Products by one constant from bank-conflict-free window tables in shared memory.
//
// Multiplication by a fixed c is GF(2)-linear, so c * a is the XOR over the W-bit windows
// a_k of a of T[k][a_k] = c * (a_k x^(W k)). A 16-byte lookup (ld.shared.v4) is served eight
// lanes at a time, and eight lanes that look up data-dependent entries of one table collide
// in the sixteen-byte bank groups: the byte tables of field.cuh spend 55-60 % of their shared
// wavefronts on that. Here every entry is stored eight times, once per bank group, and a lane
// reads the copy of its own group (lane mod 8): no lookup ever conflicts, at eight times the
// table size, which smaller windows make up for. Products per second by a block constant,
// GB300, 152 SMs (chains of products, all by table / one in four by split multiply):
//   byte table, 16 lookups, 64 KB, three blocks an SM      5.8e10 / 7.5e10 (half split)
//   W = 4, 32 lookups,  64 KB, three 256-thread blocks     7.2e10 / 8.4e10
//   W = 5, 26 lookups, 101 KB, two 256-thread blocks       9.1e10 / 9.7e10
//   W = 6, 22 lookups, 169 KB, one 512-thread block       1.07e11 / 1.11e11
// The lookups alone need 2.75 (W = 6), 3.25 and 4 cycles of the SM's shared-memory pipe a
// product, which is what the all-table figures reach.
#pragma once
#include "field.cuh"

namespace flock {
namespace gpu {

template <int W>
struct WinTable {
  static constexpr int WINDOWS = (128 + W - 1) / W;
  static constexpr int TOP_BITS = 128 - W * (WINDOWS - 1);  // bits of the last window
  static constexpr int ENTRIES = (WINDOWS - 1) * (1 << W) + (1 << TOP_BITS);
  static constexpr int BYTES = ENTRIES * 128;  // eight 16-byte copies an entry
};

// c x^i for i < 128: the 256-bit shift, reduced.
__device__ __forceinline__ F128d mul_by_power(F128d c, uint32_t i) {
  const uint32_t s = i & 63;
  const uint64_t w0 = c.lo << s, w1 = (c.hi << s) | (s ? c.lo >> (64 - s) : 0), w2 = s ? c.hi >> (64 - s) : 0;
  return i < 64 ? ghash_reduce(w0, w1, w2, 0) : ghash_reduce(0, w0, w1, w2);
}

// Fills the table of c at T (16-byte aligned, WinTable<W>::BYTES). Every thread of the block
// calls this (blockDim.x a multiple of 32); the caller puts a block barrier before the first
// lookup, and one between the last lookup of the previous contents and this call. Eight
// consecutive threads share a part of one window: lane r forms the image c x^(W k + r), the
// eight exchange them by shuffles, and each walks the part's values in Gray-code order, one
// XOR and one store into its own bank group per value (no lookups, no conflicts).
template <int W>
__device__ __forceinline__ void build_win_table(F128d c, char* T) {
  using WT = WinTable<W>;
  constexpr int LOW = W - 1;  // walked bits; the part number is the window's top bit
  constexpr int ITEMS = WT::WINDOWS * 2;
  const uint32_t r = threadIdx.x & 7, teams = blockDim.x >> 3;
  for (uint32_t it0 = 0; it0 < ITEMS; it0 += teams) {
    const uint32_t it = it0 + (threadIdx.x >> 3);
    const uint32_t k = it >> 1, part = it & 1;
    const uint32_t p = W * k + r;
    const F128d mine = (it < ITEMS && p < 128) ? mul_by_power(c, p) : f128_zero();
    F128d E[W];
#pragma unroll
    for (int b = 0; b < W; ++b) {
      E[b].lo = __shfl_sync(0xffffffffu, mine.lo, b, 8);
      E[b].hi = __shfl_sync(0xffffffffu, mine.hi, b, 8);
    }
    const uint32_t limit = k == WT::WINDOWS - 1 ? 1u << WT::TOP_BITS : 1u << W;  // values of this window
    if (it < ITEMS && (part << LOW) < limit) {
      char* o = T + ((k << W) + (part << LOW)) * 128 + r * 16;
      F128d acc = part ? E[LOW] : f128_zero();
      *reinterpret_cast<F128d*>(o) = acc;
#pragma unroll
      for (int g = 1; g < (1 << LOW); ++g) {
        int b = 0;
        while (!((g >> b) & 1)) ++b;  // the bit that the Gray code flips
        acc += E[b];
        const int v = g ^ (g >> 1);
        if ((uint32_t)v < limit) *reinterpret_cast<F128d*>(o + v * 128) = acc;
      }
    }
  }
}

// The table of any GF(2)-linear map of the low `BITS` bits of a word from the map's images
// E[i] of x^i (readable by every thread: shared or global memory), the same walk.
template <int W, int BITS>
struct WinMap {
  static constexpr int WINDOWS = (BITS + W - 1) / W;
  static constexpr int TOP_BITS = BITS - W * (WINDOWS - 1);
  static constexpr int ENTRIES = (WINDOWS - 1) * (1 << W) + (1 << TOP_BITS);
  static constexpr int BYTES = ENTRIES * 128;
};
// `teams` groups of eight threads share the work; this thread's is `team` (whole warps call).
template <int W, int BITS>
__device__ __forceinline__ void build_win_map(const F128d* E, char* T, uint32_t team, uint32_t teams) {
  using WM = WinMap<W, BITS>;
  constexpr int LOW = W - 1;
  constexpr int ITEMS = WM::WINDOWS * 2;
  const uint32_t r = threadIdx.x & 7;
  for (uint32_t it = team; it < ITEMS; it += teams) {
    const uint32_t k = it >> 1, part = it & 1;
    F128d e[W];
#pragma unroll
    for (int b = 0; b < W; ++b) e[b] = W * k + b < BITS ? E[W * k + b] : f128_zero();
    const uint32_t limit = k == WM::WINDOWS - 1 ? 1u << WM::TOP_BITS : 1u << W;
    if ((part << LOW) < limit) {
      char* o = T + ((k << W) + (part << LOW)) * 128 + r * 16;
      F128d acc = part ? e[LOW] : f128_zero();
      *reinterpret_cast<F128d*>(o) = acc;
#pragma unroll
      for (int g = 1; g < (1 << LOW); ++g) {
        int b = 0;
        while (!((g >> b) & 1)) ++b;
        acc += e[b];
        const int v = g ^ (g >> 1);
        if ((uint32_t)v < limit) *reinterpret_cast<F128d*>(o + v * 128) = acc;
      }
    }
  }
}
// acc += the map's value at the 64-bit x.
template <int W>
__device__ __forceinline__ void add_win_map64(F128d& acc, uint64_t x64, const char* T, uint32_t lane) {
  using WM = WinMap<W, 64>;
  const uint32_t x0 = (uint32_t)x64, x1 = (uint32_t)(x64 >> 32);
  uint32_t r0 = (uint32_t)acc.lo, r1 = (uint32_t)(acc.lo >> 32), r2 = (uint32_t)acc.hi, r3 = (uint32_t)(acc.hi >> 32);
#pragma unroll
  for (int k = 0; k < WM::WINDOWS; ++k) {
    const int o = W * k, s = o & 31;
    const int bits = k == WM::WINDOWS - 1 ? WM::TOP_BITS : W;
    uint32_t v;
    if (s + bits <= 32) v = s >= 7 ? (o < 32 ? x0 : x1) >> (s - 7) : (o < 32 ? x0 : x1) << (7 - s);
    else v = __funnelshift_r(x0, x1, s - 7);
    v = (v & (((1u << bits) - 1) << 7)) | lane;
    const uint4 t = *reinterpret_cast<const uint4*>(T + k * ((1 << W) * 128) + v);
    r0 ^= t.x;
    r1 ^= t.y;
    r2 ^= t.z;
    r3 ^= t.w;
  }
  acc = f128(r0 | ((uint64_t)r1 << 32), r2 | ((uint64_t)r3 << 32));
}

// This thread's bank group: the offset its lookups add.
__device__ __forceinline__ uint32_t win_lane() { return (threadIdx.x & 7) << 4; }

// a * c from the table of c. T: the shared array itself (with a constant offset), so that the
// windows' bases become immediate offsets of the loads.
template <int W>
__device__ __forceinline__ F128d mul_win(F128d a, const char* T, uint32_t lane) {
  using WT = WinTable<W>;
  const uint32_t x[4] = {(uint32_t)a.lo, (uint32_t)(a.lo >> 32), (uint32_t)a.hi, (uint32_t)(a.hi >> 32)};
  uint32_t r0 = 0, r1 = 0, r2 = 0, r3 = 0;
#pragma unroll
  for (int k = 0; k < WT::WINDOWS; ++k) {
    const int o = W * k, w = o >> 5, s = o & 31;
    const int bits = k == WT::WINDOWS - 1 ? WT::TOP_BITS : W;
    // the window's bits moved to bit 7 (entries are 128 bytes apart)
    uint32_t v;
    if (s + bits <= 32) v = s >= 7 ? x[w] >> (s - 7) : x[w] << (7 - s);
    else v = __funnelshift_r(x[w], x[w + 1 < 4 ? w + 1 : 3], s - 7);  // a window across two words: s > 7
    v = (v & (((1u << bits) - 1) << 7)) | lane;
    const uint4 t = *reinterpret_cast<const uint4*>(T + k * ((1 << W) * 128) + v);
    r0 ^= t.x;
    r1 ^= t.y;
    r2 ^= t.z;
    r3 ^= t.w;
  }
  return f128(r0 | ((uint64_t)r1 << 32), r2 | ((uint64_t)r3 << 32));
}

}  // namespace gpu
}  // namespace flock
