// Witness generation on the device: a block's z, a = A_0 z and b = B_0 z bits straight into the
// batch-major layout (word (c << nu) + instance holds bits [128 c, 128 c + 128) of the instance's
// block; crates/flock-prover/src/r1cs_hashes/common.rs:456-585). Threads of a warp are
// consecutive instances, so every 16-byte chunk store of a warp is one coalesced 512-byte line,
// and every word is written exactly once (gaps between fields as zeros).
//
// BLAKE3 and SHA-256 split an instance's chunks over the grid's y: a thread runs the hash from its
// input in registers (cheap: the whole compression is about 800 or 2500 instructions) and emits only
// the fields of its own chunk range; a chunk that spans two ranges is emitted by one of them,
// which forms the other's few fields too. One thread per instance, which this replaced, was a
// serial chain of all fields with the state in local memory: 69 us (BLAKE3) and 140 us (SHA-256)
// whatever the batch up to 2^13.
//
// Per-hash field semantics follow build_group_batch_major:
//   BLAKE3   blake3.rs:1929-2040      SHA-256  sha2.rs:1743-1850      Keccak  keccak.rs:565-640
#include "kernels.h"
#include <mutex>
#include "../host/r1cs_blake3.h"
#include "../host/r1cs_sha2.h"
#include "../host/r1cs_keccak.h"

namespace flock {
namespace gpu {

// The bits of consecutive fields of z, a and b, 32 at a time: complete words shift through four
// registers, a complete chunk in [lo, hi) is stored. Bit positions only grow; they are the same
// for all instances, so every branch on them is uniform.
struct FieldStream {
  uint4 *z, *a, *b;  // this instance's word of chunk 0
  uint32_t nu, lo, hi, word, fill;  // the open word and the bits in it
  uint32_t zc, ac, bc;
  uint4 zv, av, bv;

  // The first field put is at bit `pos`, each later one where the one before ended.
  __device__ __forceinline__ void init(uint4* zz, uint4* aa, uint4* bb, uint32_t nu_, uint32_t inst, uint32_t pos,
                                       uint32_t lo_, uint32_t hi_) {
    z = zz + inst; a = aa + inst; b = bb + inst;
    nu = nu_; lo = lo_; hi = hi_;
    word = pos >> 5;
    fill = pos & 31;
    zc = ac = bc = 0;
    zv = av = bv = make_uint4(0, 0, 0, 0);
  }
  __device__ __forceinline__ void step() {
    zv = make_uint4(zv.y, zv.z, zv.w, zc);
    av = make_uint4(av.y, av.z, av.w, ac);
    bv = make_uint4(bv.y, bv.z, bv.w, bc);
    zc = ac = bc = 0;
    if ((++word & 3) == 0) {
      const uint32_t c = (word >> 2) - 1;
      if (c >= lo && c < hi) {
        const size_t w = (size_t)c << nu;
        z[w] = zv; a[w] = av; b[w] = bv;
      }
    }
  }
  // The next n bits (1 <= n <= 32).
  __device__ __forceinline__ void put(uint32_t n, uint32_t zx, uint32_t ax, uint32_t bx) {
    zc |= zx << fill; ac |= ax << fill; bc |= bx << fill;
    const uint32_t sh = 32 - fill;  // the bits from here on are the next word's
    fill += n;
    if (fill >= 32) {
      step();
      zc = __funnelshift_rc(zx, 0, sh); ac = __funnelshift_rc(ax, 0, sh); bc = __funnelshift_rc(bx, 0, sh);
      fill -= 32;
    }
  }
  __device__ __forceinline__ void put(uint32_t v) { put(32, v, v, 0xFFFFFFFFu); }
  // Complete the chunks below hi with zeros.
  __device__ __forceinline__ void finish() {
    while (word < hi * 4) step();
  }
};
__host__ __device__ constexpr uint32_t chunk_up(uint32_t bit) { return (bit + 127) / 128; }

__device__ __forceinline__ uint32_t rotr32d(uint32_t x, int n) { return __funnelshift_r(x, x, n); }

struct Add3 { uint32_t sum, m0, m1, m2, r0, r1, r2; };
__device__ __forceinline__ Add3 fadd3(uint32_t x, uint32_t y, uint32_t m) {
  uint32_t xm = x ^ m, ym = y ^ m, w = xm & ym, p = x ^ y ^ m, bw = (w ^ m) << 1;
  uint32_t sum = p + bw, cin = sum ^ p ^ bw, rl = p ^ cin, rr = bw ^ cin;
  Add3 o;
  o.sum = sum;
  o.m0 = xm & 0x7FFFFFFFu; o.m1 = ym & 0x7FFFFFFFu; o.m2 = w & 0x7FFFFFFFu;
  o.r0 = (rl >> 1) & 0x3FFFFFFFu; o.r1 = (rr >> 1) & 0x3FFFFFFFu; o.r2 = ((rl & rr) >> 1) & 0x3FFFFFFFu;
  return o;
}
struct Add2 { uint32_t sum, l, r, c; };
__device__ __forceinline__ Add2 add2(uint32_t x, uint32_t y) {
  uint32_t s = x + y, cin = s ^ x ^ y, l = (x ^ cin) & 0x7FFFFFFFu, r = (y ^ cin) & 0x7FFFFFFFu;
  Add2 o; o.sum = s; o.l = l; o.r = r; o.c = l & r;
  return o;
}

// ------------------------------------------------------------------------ BLAKE3
__constant__ uint32_t B3_IV_C[8] = {0x6a09e667, 0xbb67ae85, 0x3c6ef372, 0xa54ff53a,
                                    0x510e527f, 0x9b05688c, 0x1f83d9ab, 0x5be0cd19};
__constant__ uint32_t B3_GBASE[57];

__device__ __forceinline__ void b3_g(uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d, uint32_t mx, uint32_t my) {
  a += b + mx; d = rotr32d(d ^ a, 16);
  c += d;      b = rotr32d(b ^ c, 12);
  a += b + my; d = rotr32d(d ^ a, 8);
  c += d;      b = rotr32d(b ^ c, 7);
}
__device__ __forceinline__ void b3_permute(uint32_t (&m)[16]) {
  constexpr int P[16] = {2, 6, 3, 10, 7, 0, 4, 13, 1, 11, 12, 5, 9, 14, 15, 8};
  uint32_t t[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) t[i] = m[P[i]];
#pragma unroll
  for (int i = 0; i < 16; ++i) m[i] = t[i];
}
__device__ __forceinline__ void b3_round(uint32_t (&s)[16], const uint32_t (&m)[16]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) b3_g(s[i], s[4 + i], s[8 + i], s[12 + i], m[2 * i], m[2 * i + 1]);
#pragma unroll
  for (int i = 0; i < 4; ++i)
    b3_g(s[i], s[4 + (i + 1) % 4], s[8 + (i + 2) % 4], s[12 + (i + 3) % 4], m[8 + 2 * i], m[9 + 2 * i]);
}
// Row `ROW` of the state rotated by N places.
template <int ROW, int N>
__device__ __forceinline__ void b3_rotate(uint32_t (&s)[16]) {
  uint32_t t[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) t[i] = s[4 * ROW + (i + N) % 4];
#pragma unroll
  for (int i = 0; i < 4; ++i) s[4 * ROW + i] = t[i];
}
// The G of column 0 with message words m[0], m[1] and its fields; then the next column and the next
// words move to the front, so that one copy of this code serves every G (unrolled over a
// round's eight it was bound by instruction fetches: each line of it ran twice).
__device__ __forceinline__ void b3_emit(FieldStream& W, uint32_t (&s)[16], uint32_t (&m)[16], uint32_t g) {
  const Add3 f1 = fadd3(s[0], s[4], m[0]);
  W.put(31, f1.m2, f1.m0, f1.m1);
  W.put(30, f1.r2, f1.r0, f1.r1);
  const uint32_t d1 = rotr32d(s[12] ^ f1.sum, 16);
  const Add2 p = add2(s[8], d1);
  // the first four G's add to constants: the rows below the constant's lowest one bit fall away
  const uint32_t t = g < 2 ? 1 : g < 4 ? 2 : 0;
  W.put(31 - t, p.c >> t, p.l >> t, p.r >> t);
  const uint32_t b1 = rotr32d(s[4] ^ p.sum, 12);
  const Add3 f2 = fadd3(f1.sum, b1, m[1]);
  W.put(31, f2.m2, f2.m0, f2.m1);
  W.put(30, f2.r2, f2.r0, f2.r1);
  const uint32_t d2 = rotr32d(d1 ^ f2.sum, 8);
  const Add2 p2 = add2(p.sum, d2);
  W.put(31, p2.c, p2.l, p2.r);
  s[0] = f2.sum;
  s[4] = rotr32d(b1 ^ p2.sum, 7);
  s[8] = p2.sum;
  s[12] = d2;
  b3_rotate<0, 1>(s); b3_rotate<1, 1>(s); b3_rotate<2, 1>(s); b3_rotate<3, 1>(s);
  const uint32_t u0 = m[0], u1 = m[1];
#pragma unroll
  for (int i = 0; i < 14; ++i) m[i] = m[i + 2];
  m[14] = u0;
  m[15] = u1;
}

// Part 0: the input and output words; part y >= 1: the G's of round y - 1, from the chunk that the
// round begins in the middle of (its own fields fill the one before) to the first chunk past it.
constexpr uint32_t B3_PARTS = 8;
__global__ void __launch_bounds__(64, 8)
witness_blake3_kernel(const b3r1cs::Compression* __restrict__ in, uint32_t n_inst, uint32_t nu, uint4* z, uint4* a,
                      uint4* b, uint32_t used_chunks) {
  const uint32_t o = blockIdx.x * blockDim.x + threadIdx.x, part = blockIdx.y;
  if (o >= n_inst) return;
  static_assert(b3r1cs::CV_BASE == 0 && b3r1cs::OUT_LO_BASE == 256 && b3r1cs::M_BASE == 512 &&
                b3r1cs::T_LO_BASE == 1024 && b3r1cs::OUT_HI_BASE == 1152 && b3r1cs::GS_BASE == 1408, "no gaps");
  uint32_t cv[8], m[16], m0[16], s[16];
#pragma unroll
  for (int i = 0; i < 8; ++i) s[i] = cv[i] = in[o].cv[i];
#pragma unroll
  for (int i = 0; i < 16; ++i) m[i] = m0[i] = in[o].m[i];
#pragma unroll
  for (int i = 0; i < 4; ++i) s[8 + i] = B3_IV_C[i];
  const uint64_t counter = in[o].counter;
  s[12] = (uint32_t)counter; s[13] = (uint32_t)(counter >> 32); s[14] = in[o].block_len; s[15] = in[o].flags;
  const uint32_t tail[4] = {s[12], s[13], s[14], s[15]};
  FieldStream W;
  if (part == 0) {
    for (int r = 0; r < 7; ++r) {
      b3_round(s, m);
      b3_permute(m);
    }
    W.init(z, a, b, nu, o, 0, 0, b3r1cs::GS_BASE / 128);
    static_assert(b3r1cs::GS_BASE % 128 == 0, "the first G begins a chunk");
#pragma unroll
    for (int w = 0; w < 8; ++w) W.put(cv[w]);
#pragma unroll
    for (int w = 0; w < 8; ++w) W.put(s[w] ^ s[w + 8]);
#pragma unroll
    for (int i = 0; i < 16; ++i) W.put(m0[i]);
#pragma unroll
    for (int i = 0; i < 4; ++i) W.put(tail[i]);
#pragma unroll
    for (int w = 0; w < 8; ++w) W.put(s[w + 8] ^ cv[w]);
    W.finish();
    return;
  }
  const uint32_t r0 = part - 1;
  for (uint32_t r = 0; r < r0; ++r) {
    b3_round(s, m);
    b3_permute(m);
  }
  const uint32_t base = B3_GBASE[8 * r0], end = B3_GBASE[8 * r0 + 8];
  W.init(z, a, b, nu, o, base, chunk_up(base), part == B3_PARTS - 1 ? used_chunks : chunk_up(end));
  // the round's eight G's, and the next round's first for the last chunk
  const uint32_t last = min(8 * r0 + 9, 56u);
#pragma unroll 1
  for (uint32_t g = 8 * r0; g < last; ++g) {
    b3_emit(W, s, m, g);
    if ((g & 7) == 3) { b3_rotate<1, 1>(s); b3_rotate<2, 2>(s); b3_rotate<3, 3>(s); }
    if ((g & 7) == 7) {
      b3_rotate<1, 3>(s); b3_rotate<2, 2>(s); b3_rotate<3, 1>(s);
      b3_permute(m);
    }
  }
  if (part == B3_PARTS - 1) W.put(1, 1, 1, 1);
  W.finish();
}

// ------------------------------------------------------------------------ SHA-256
__constant__ uint32_t S2_K[64];
__constant__ uint32_t S2_ROUND_BASE[65];

__device__ __forceinline__ uint32_t bs0(uint32_t x) { return rotr32d(x, 2) ^ rotr32d(x, 13) ^ rotr32d(x, 22); }
__device__ __forceinline__ uint32_t bs1(uint32_t x) { return rotr32d(x, 6) ^ rotr32d(x, 11) ^ rotr32d(x, 25); }
__device__ __forceinline__ uint32_t ss0(uint32_t x) { return rotr32d(x, 7) ^ rotr32d(x, 18) ^ (x >> 3); }
__device__ __forceinline__ uint32_t ss1(uint32_t x) { return rotr32d(x, 17) ^ rotr32d(x, 19) ^ (x >> 10); }

struct Add4 { uint32_t sum, m1[3], m2[3], r[3]; };
__device__ __forceinline__ Add4 fadd4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  uint32_t xz = x ^ z, yz = y ^ z, w1 = xz & yz, p1 = x ^ y ^ z, b1 = (w1 ^ z) << 1;
  uint32_t pw = p1 ^ w, bw = b1 ^ w, w2 = pw & bw, p2 = p1 ^ b1 ^ w, b2 = (w2 ^ w) << 1;
  uint32_t sum = p2 + b2, cin = sum ^ p2 ^ b2, rl = p2 ^ cin, rr = b2 ^ cin;
  Add4 o;
  o.sum = sum;
  o.m1[0] = xz & 0x7FFFFFFFu; o.m1[1] = yz & 0x7FFFFFFFu; o.m1[2] = w1 & 0x7FFFFFFFu;
  o.m2[0] = pw & 0x7FFFFFFFu; o.m2[1] = bw & 0x7FFFFFFFu; o.m2[2] = w2 & 0x7FFFFFFFu;
  o.r[0] = (rl >> 1) & 0x3FFFFFFFu; o.r[1] = (rr >> 1) & 0x3FFFFFFFu; o.r[2] = ((rl & rr) >> 1) & 0x3FFFFFFFu;
  return o;
}

__device__ __forceinline__ void put_add4(FieldStream& R, const Add4& p) {
  R.put(31, p.m1[2], p.m1[0], p.m1[1]);
  R.put(31, p.m2[2], p.m2[0], p.m2[1]);
  R.put(30, p.r[2], p.r[0], p.r[1]);
}
// The compression at round r: w[i] holds W[r + i], st the registers a .. h going in. The loops that
// emit many fields a round hold one round (unrolled over the sixteen of a window they were bound
// by instruction fetches), the others four.
struct Sha2Run {
  uint32_t st[8], w[16];
  __device__ __forceinline__ void load(const s2r1cs::Compression* in) {
#pragma unroll
    for (int i = 0; i < 8; ++i) st[i] = in->h[i];
#pragma unroll
    for (int i = 0; i < 16; ++i) w[i] = in->w[i];
  }
  // The terms of W[r + 16] in the fields' order.
  __device__ __forceinline__ Add4 sched_terms() const { return fadd4(ss1(w[14]), ss0(w[1]), w[9], w[0]); }
  __device__ __forceinline__ void sched() {
    const uint32_t next = ss1(w[14]) + ss0(w[1]) + w[9] + w[0];
#pragma unroll
    for (int i = 0; i < 15; ++i) w[i] = w[i + 1];
    w[15] = next;
  }
  __device__ __forceinline__ void round(uint32_t r) {
    const uint32_t t1 = st[7] + bs1(st[4]) + ((st[4] & st[5]) ^ (~st[4] & st[6])) + S2_K[r] + w[0];
    const uint32_t t2 = bs0(st[0]) + ((st[0] & st[1]) ^ (st[0] & st[2]) ^ (st[1] & st[2]));
    st[7] = st[6]; st[6] = st[5]; st[5] = st[4]; st[4] = st[3] + t1;
    st[3] = st[2]; st[2] = st[1]; st[1] = st[0]; st[0] = t1 + t2;
    sched();
  }
  __device__ __forceinline__ void rounds(uint32_t r0, uint32_t r1) {
#pragma unroll 4
    for (uint32_t r = r0; r < r1; ++r) round(r);
  }
  // The additions of round r.
  __device__ __forceinline__ void emit_round(FieldStream& R, uint32_t r) const {
    const uint32_t k = S2_K[r];
    const uint32_t ch_out = (st[4] & (st[5] ^ st[6])) ^ st[6];
    const uint32_t maj_out = ((st[1] ^ st[0]) & (st[2] ^ st[0])) ^ st[0];
    const uint32_t t = __ffs(k);  // trailing_zeros(k) + 1
    const Add2 kp = add2(k, st[7]);
    const Add4 t1 = fadd4(kp.sum, bs1(st[4]), ch_out, w[0]);
    put_add4(R, t1);
    const Add3 an = fadd3(t1.sum, bs0(st[0]), maj_out);
    R.put(31, an.m2, an.m0, an.m1);
    R.put(30, an.r2, an.r0, an.r1);
    const Add2 en = add2(st[3], t1.sum);
    R.put(31, en.c, en.l, en.r);
    R.put(31 - t, kp.c >> t, kp.l >> t, kp.r >> t);
  }
};

// Parts: 0 the input and output words, 1 and 2 the ch and maj products, 3 .. 6 sixteen rounds'
// additions each, 7 the schedule, 8 and 9 the e and a words with the output additions. A part starts with
// the last fields of the one before where its first chunk begins in them.
constexpr uint32_t S2_PARTS = 10;
template <uint32_t PART>
__device__ __forceinline__ void sha2_part(const s2r1cs::Compression* in, uint32_t nu, uint32_t o, uint4* z, uint4* a,
                                          uint4* b, uint32_t used_chunks) {
  using namespace s2r1cs;
  static_assert(H_BASE == 0 && H_OUT_BASE == 256 && M_BASE == 512 && CH_AND_BASE == 1024 && MAJ_AND_BASE == 3072 &&
                ROUND_CARRY_BASE == 5120, "whole chunks, no gaps");
  Sha2Run x;
  FieldStream R;
  x.load(in);
  if constexpr (PART == 0) {
    x.rounds(0, 64);
    R.init(z, a, b, nu, o, 0, 0, CH_AND_BASE / 128);
#pragma unroll
    for (int w = 0; w < 8; ++w) R.put(in->h[w]);
#pragma unroll
    for (int w = 0; w < 8; ++w) R.put(x.st[w] + in->h[w]);
#pragma unroll
    for (int i = 0; i < 16; ++i) R.put(in->w[i]);
  } else if constexpr (PART <= 2) {
    constexpr uint32_t base = PART == 1 ? CH_AND_BASE : MAJ_AND_BASE;
    R.init(z, a, b, nu, o, base, base / 128, base / 128 + 16);
#pragma unroll 4
    for (uint32_t r = 0; r < 64; ++r) {
      const uint32_t l = PART == 1 ? x.st[4] : x.st[1] ^ x.st[0];
      const uint32_t m = PART == 1 ? x.st[5] ^ x.st[6] : x.st[2] ^ x.st[0];
      R.put(32, l & m, l, m);
      x.round(r);
    }
  } else if constexpr (PART <= 6) {
    constexpr uint32_t r0 = 16 * (PART - 3);
    const uint32_t base = S2_ROUND_BASE[r0];
    x.rounds(0, r0);
    R.init(z, a, b, nu, o, base, chunk_up(base), chunk_up(S2_ROUND_BASE[r0 + 16]));
    // the next round too, for the last chunk
#pragma unroll 1
    for (uint32_t r = r0; r < r0 + (r0 < 48 ? 17 : 16); ++r) {
      x.emit_round(R, r);
      x.round(r);
    }
    if constexpr (r0 == 48) {  // the chunk ends in the first two additions of the schedule
      x.load(in);
#pragma unroll 1
      for (int i = 0; i < 2; ++i) {
        put_add4(R, x.sched_terms());
        x.sched();
      }
    }
  } else if constexpr (PART == 7) {
    R.init(z, a, b, nu, o, SCHED_CARRY_BASE, chunk_up(SCHED_CARRY_BASE), E_NEW_BASE / 128);
#pragma unroll 1
    for (uint32_t t = 16; t < 64; ++t) {
      put_add4(R, x.sched_terms());
      x.sched();
    }
  } else {
    // word i of the region is register a or e after round 2 i + 1
    constexpr uint32_t base = PART == 8 ? E_NEW_BASE : A_NEW_BASE, first = base / 128;
    if constexpr (PART == 8) {
      // the first chunk begins in the last additions of the schedule, W[62] and W[63]
#pragma unroll 4
      for (uint32_t t = 16; t < 62; ++t) x.sched();
      constexpr uint32_t last = SCHED_CARRY_BASE + 46 * SCHED_ADD_BITS;
      static_assert(last / 128 <= first && last + 2 * SCHED_ADD_BITS == base, "two additions reach into the chunk");
      R.init(z, a, b, nu, o, last, first, A_NEW_BASE / 128);
#pragma unroll 1
      for (uint32_t t = 62; t < 64; ++t) {
        put_add4(R, x.sched_terms());
        x.sched();
      }
    } else {
      // the first chunk begins in the e word of the last round
      x.rounds(0, 64);
      R.init(z, a, b, nu, o, base - 32, first, used_chunks);
      R.put(x.st[4]);
    }
    x.load(in);
#pragma unroll 2
    for (uint32_t r = 0; r < 64; r += 2) {
      x.round(r);
      x.round(r + 1);
      R.put(x.st[PART == 8 ? 4 : 0]);
    }
    if constexpr (PART == 9) {
#pragma unroll
      for (int w = 0; w < 8; ++w) {
        const Add2 oc = add2(x.st[w], in->h[w]);
        R.put(31, oc.c, oc.l, oc.r);
      }
      R.put(1, 1, 1, 1);
    }
  }
  R.finish();
}
__global__ void __launch_bounds__(64, 8)
witness_sha2_kernel(const s2r1cs::Compression* __restrict__ in, uint32_t n_inst, uint32_t nu, uint4* z, uint4* a,
                    uint4* b, uint32_t used_chunks) {
  const uint32_t o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= n_inst) return;
  in += o;
  switch (blockIdx.y) {
    case 0: sha2_part<0>(in, nu, o, z, a, b, used_chunks); break;
    case 1: sha2_part<1>(in, nu, o, z, a, b, used_chunks); break;
    case 2: sha2_part<2>(in, nu, o, z, a, b, used_chunks); break;
    case 3: sha2_part<3>(in, nu, o, z, a, b, used_chunks); break;
    case 4: sha2_part<4>(in, nu, o, z, a, b, used_chunks); break;
    case 5: sha2_part<5>(in, nu, o, z, a, b, used_chunks); break;
    case 6: sha2_part<6>(in, nu, o, z, a, b, used_chunks); break;
    case 7: sha2_part<7>(in, nu, o, z, a, b, used_chunks); break;
    case 8: sha2_part<8>(in, nu, o, z, a, b, used_chunks); break;
    default: sha2_part<9>(in, nu, o, z, a, b, used_chunks); break;
  }
}

// ------------------------------------------------------------------------ Keccak-f[1600]
__constant__ uint64_t KC_RC[24];
__device__ __forceinline__ uint64_t rotl64d(uint64_t v, uint32_t r) { return r ? (v << r) | (v >> (64 - r)) : v; }

// One thread per instance; the 64-bit words of a block leave in pairs, one 16-byte store a chunk, and
// the rotations are compile-time
// (2^18 instances: 1.14 -> 0.63 ms, 0.62 ms of HBM writes at the measured rate).
__global__ void witness_keccak_kernel(const uint64_t* __restrict__ in, uint32_t n_inst, uint32_t nu,
                                      ulonglong2* z, ulonglong2* a, ulonglong2* b, uint32_t used_words) {
  uint32_t o = blockIdx.x * blockDim.x + threadIdx.x;
  if (o >= n_inst) return;
  // input words -> Keccak lanes: input bit j is bit j / 25 of lane j % 25. The input words
  // are loaded once and every index below is a compile-time constant (fully unrolled), so
  // the lanes stay in registers.
  uint64_t iw[25];
#pragma unroll
  for (int i = 0; i < 25; ++i) iw[i] = in[(size_t)o * 25 + i];
  uint64_t st[25];
#pragma unroll
  for (int l = 0; l < 25; ++l) {
    uint64_t v = 0;
#pragma unroll
    for (int k = 0; k < 64; ++k) {
      const int j = 25 * k + l;
      v |= ((iw[j >> 6] >> (j & 63)) & 1ull) << k;
    }
    st[l] = v;
  }
  // words w (even: held back) and w + 1 of the block are chunk w / 2
  uint64_t hz, ha, hb;
  auto put = [&](uint32_t w, uint64_t zv, uint64_t av, uint64_t bv) {
    if (w & 1) {
      const size_t idx = (((size_t)(w >> 1)) << nu) + o;
      z[idx] = make_ulonglong2(hz, zv);
      a[idx] = make_ulonglong2(ha, av);
      b[idx] = make_ulonglong2(hb, bv);
    } else {
      hz = zv; ha = av; hb = bv;
    }
  };
#pragma unroll
  for (int w = 0; w < 32; ++w) put(w, w < 25 ? st[w] : 0, w < 25 ? st[w] : 0, w < 25 ? ~0ull : 0);
  // the constant, then the rounds' products from word 65 on: two rounds are 25 chunks
  static_assert(kr1cs::Z_CONST == 64 * 64 && kr1cs::T_PACKED_BIT_BASE == 65 * 64, "the products follow the constant");
  put(64, 1, 1, 1);
  for (uint32_t r2 = 0; r2 < 24; r2 += 2) {
#pragma unroll
    for (uint32_t k = 0; k < 2; ++k) {
      const uint32_t r = r2 + k;
      uint64_t th[25], bs[25], cc[5];
#pragma unroll
      for (int x = 0; x < 5; ++x) cc[x] = st[x] ^ st[x + 5] ^ st[x + 10] ^ st[x + 15] ^ st[x + 20];
#pragma unroll
      for (int i = 0; i < 25; ++i) th[i] = st[i] ^ cc[(i % 5 + 4) % 5] ^ rotl64d(cc[(i % 5 + 1) % 5], 1);
#pragma unroll
      for (int y = 0; y < 5; ++y)
#pragma unroll
        for (int x = 0; x < 5; ++x) {
          constexpr uint32_t RHO[25] = {0, 1, 62, 28, 27, 36, 44, 6, 55, 20, 3, 10, 43,
                                        25, 39, 41, 45, 15, 21, 8, 18, 2, 61, 56, 14};  // of lane a + 5 b
          const int src = (x + 3 * y) % 5 + 5 * x;
          bs[x + 5 * y] = rotl64d(th[src], RHO[src]);
        }
      const uint32_t tb = 65 + r2 * 25;  // odd
#pragma unroll
      for (int y = 0; y < 5; ++y)
#pragma unroll
        for (int x = 0; x < 5; ++x) {
          const uint64_t b1 = bs[(x + 1) % 5 + 5 * y], b2 = bs[(x + 2) % 5 + 5 * y], t = (~b1) & b2;
          const uint32_t i = k * 25 + x + 5 * y;  // word tb + i is the odd one of its chunk for even i
          if (i & 1) { hz = t; ha = ~b1; hb = b2; }
          else put((tb + i) | 1, t, ~b1, b2);
          st[x + 5 * y] = bs[x + 5 * y] ^ t;
        }
      st[0] ^= KC_RC[r];
    }
  }
  const uint32_t end = 65 + 24 * 25;  // odd: its chunk holds the last product
  if (end < used_words) put(end, 0, 0, 0);
  for (uint32_t w = end + 1; w < used_words; ++w) put(w, 0, 0, 0);
#pragma unroll
  for (int w = 0; w < 32; ++w) put(32 + w, w < 25 ? st[w] : 0, w < 25 ? st[w] : 0, w < 25 ? ~0ull : 0);
}

// ------------------------------------------------------------------------ launchers
void upload_witness_constants() {
  // module constants are per device
  static std::mutex mu;
  static bool done[MAX_DEVICES] = {};
  int dev = 0;
  CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= MAX_DEVICES) throw std::runtime_error("device index out of range");
  std::lock_guard<std::mutex> g(mu);
  if (done[dev]) return;
  CUDA_OK(cudaMemcpyToSymbol(B3_GBASE, b3r1cs::G_BASE.v, sizeof(uint32_t) * 57));
  CUDA_OK(cudaMemcpyToSymbol(S2_K, Sha256::K, sizeof(uint32_t) * 64));
  CUDA_OK(cudaMemcpyToSymbol(S2_ROUND_BASE, s2r1cs::ROUND_BASE.v, sizeof(uint32_t) * 65));
  CUDA_OK(cudaMemcpyToSymbol(KC_RC, kr1cs::RC, sizeof(uint64_t) * 24));
  // the copies above may still be in flight when they return; kernels of non-blocking
  // streams are not ordered after them
  CUDA_OK(cudaDeviceSynchronize());
  done[dev] = true;
}

void launch_witness(int hash, const void* d_inputs, uint32_t n_inst, uint32_t nu, F128d* z, F128d* a, F128d* b,
                    uint32_t used_chunks, cudaStream_t s) {
  upload_witness_constants();
  const uint32_t threads = 64, blocks = (n_inst + threads - 1) / threads;
  if (hash == 0)
    witness_blake3_kernel<<<dim3(blocks, B3_PARTS), threads, 0, s>>>((const b3r1cs::Compression*)d_inputs, n_inst, nu,
                                                                     (uint4*)z, (uint4*)a, (uint4*)b, used_chunks);
  else if (hash == 1)
    witness_sha2_kernel<<<dim3(blocks, S2_PARTS), threads, 0, s>>>((const s2r1cs::Compression*)d_inputs, n_inst, nu,
                                                                   (uint4*)z, (uint4*)a, (uint4*)b, used_chunks);
  else
    witness_keccak_kernel<<<blocks, threads, 0, s>>>((const uint64_t*)d_inputs, n_inst, nu, (ulonglong2*)z,
                                                     (ulonglong2*)a, (ulonglong2*)b, used_chunks * 2);
  LAUNCH_OK();
}

}  // namespace gpu
}  // namespace flock
