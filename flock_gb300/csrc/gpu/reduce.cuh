// Device helpers shared by the sumcheck and assist kernels: block-wide XOR reduction, split
// eq tables, in-kernel publication of a round message, the byte-table fold map and the
// jagged unrank of a union's committed stack.
#pragma once
#include "kernels.h"

namespace flock {
namespace gpu {

__device__ __forceinline__ F128d block_xor(F128d v, F128d* sh) {
  v = warp_xor(v);
  int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  F128d r = f128_zero();
  if (w == 0) {
    r = l < nw ? sh[l] : f128_zero();
    r = warp_xor(r);
  }
  return r;  // valid in thread 0
}

__device__ __forceinline__ F128d eq_at(const F128d* lo, uint32_t lo_bits, const F128d* hi, uint64_t i) {
  F128d l = lo[i & ((1ull << lo_bits) - 1)];
  return hi ? l * hi[i >> lo_bits] : l;
}

// ------------------------------------------------------------------ eq tables
// eq over n coordinates as a product over groups of four: the 16 values of each group in shared
// memory (a product tree of depth two), then an entry is a product tree over its groups. Four
// products deep for twelve coordinates, where one factor after the other is twelve, and a
// quarter of the products.
constexpr uint32_t EQ_THREADS = 256;
constexpr uint32_t EQ_MAX_GROUPS = 8;  // at most 32 coordinates
// Every thread of the block calls this; a barrier before the tables are read.
__device__ __forceinline__ void eq_sub_tables(const F128d* __restrict__ p, uint32_t n, F128d (*sub)[16]) {
  for (uint32_t i = threadIdx.x; i < EQ_MAX_GROUPS * 16; i += blockDim.x) {
    const uint32_t g = i >> 4, v = i & 15;
    if (4 * g >= n) continue;
    F128d f[4];
#pragma unroll
    for (uint32_t b = 0; b < 4; ++b) {
      f[b] = f128_one();
      if (4 * g + b < n) {
        f[b] = p[4 * g + b];
        if (!((v >> b) & 1)) f[b].lo ^= 1;
      }
    }
    sub[g][v] = mul_call(mul_call(f[0], f[1]), mul_call(f[2], f[3]));
  }
}
__device__ __forceinline__ F128d eq_from_sub(const F128d (*sub)[16], uint32_t n, uint64_t i) {
  const uint32_t groups = (n + 3) / 4;
  F128d v = f128_one();
  for (uint32_t g = 0; g < groups; g += 2) {
    F128d t = sub[g][(i >> (4 * g)) & 15];
    if (g + 1 < groups) t = mul_call(t, sub[g + 1][(i >> (4 * g + 4)) & 15]);
    v = g ? mul_call(v, t) : t;
  }
  return v;
}

// ------------------------------------------------------------------ fused publication
// Called by every block after thread 0 stored its `width` partials at part[block * width]:
// the block takes a ticket; the block that takes the last one reduces all partials (the
// other blocks' stores are visible to it after their fences and the atomic), writes the
// message to mapped memory, then the sequence number, and resets the counter. A block alone
// writes its partials out directly.
static __device__ void publish_if_last(const F128d* part, uint32_t width, const FusedPublish& pub, F128d* sh) {
  if (gridDim.x == 1) {  // the block's own partials are the message
    if (threadIdx.x == 0) {
      volatile F128d* o = pub.out;
      for (uint32_t j = 0; j < width; ++j) {
        o[j].lo = part[j].lo;
        o[j].hi = part[j].hi;
      }
      __threadfence_system();
      *(volatile uint32_t*)pub.flag = pub.seq;
    }
    return;
  }
  __shared__ uint32_t ticket;
  if (threadIdx.x == 0) {
    __threadfence();
    ticket = atomicAdd(pub.counter, 1u);
  }
  __syncthreads();
  if (ticket != gridDim.x - 1) return;
  __threadfence();
  for (uint32_t j = 0; j < width; ++j) {
    F128d acc = f128_zero();
    for (uint32_t b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
      const F128d* p = part + (uint64_t)b * width + j;
      acc += f128(__ldcg(&p->lo), __ldcg(&p->hi));
    }
    acc = block_xor(acc, sh);
    if (threadIdx.x == 0) {
      volatile F128d* o = pub.out;
      o[j].lo = acc.lo;
      o[j].hi = acc.hi;
    }
  }
  if (threadIdx.x == 0) {
    *pub.counter = 0;
    __threadfence_system();
    *(volatile uint32_t*)pub.flag = pub.seq;
  }
}

// Publication of data that the blocks wrote to mapped memory themselves: every thread of the
// block calls this after its writes; the last block to arrive sets the sequence number.
static __device__ void publish_data(const FusedPublish& pub) {
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence_system();
    if (atomicAdd(pub.counter, 1u) == gridDim.x * gridDim.y - 1) {
      *pub.counter = 0;
      __threadfence_system();
      *(volatile uint32_t*)pub.flag = pub.seq;
    }
  }
}

// ------------------------------------------------------------------ byte-table maps, jagged layout
__device__ __forceinline__ F128d fold_slot(F128d x, const F128d* tab) {
  F128d acc = f128_zero();
#pragma unroll
  for (int k = 0; k < 8; ++k) acc += tab[k * 256 + ((x.lo >> (8 * k)) & 255)];
#pragma unroll
  for (int k = 0; k < 8; ++k) acc += tab[(8 + k) * 256 + ((x.hi >> (8 * k)) & 255)];
  return acc;
}
// Jagged unrank of a union's committed stack: slot s holds dense [base, base + rows * cols),
// column-major with `rows` (the declared count) words per column, its first column at
// union chunk-column col_off.
__device__ __forceinline__ bool jagged_unrank(const JaggedSegs& g, uint64_t d, uint64_t& row, uint64_t& col) {
  for (uint32_t s = 0; s < g.n; ++s) {
    const uint64_t end = g.base[s] + g.rows[s] * g.cols[s];
    if (d >= g.base[s] && d < end) {
      const uint64_t local = d - g.base[s];
      col = g.col_off[s] + local / g.rows[s];
      row = local % g.rows[s];
      return true;
    }
  }
  return false;
}
}  // namespace gpu
}  // namespace flock
