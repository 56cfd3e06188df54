// Device SHA-256 (FIPS 180-4) for the Merkle commitments of the L0 codeword and the
// recursive Ligerito levels (leaf = SHA256(row bytes), node = SHA256(left || right);
// crates/flock-core/src/merkle.rs:205-232) and for the transcript proof-of-work search
// (SHA256(state_digest || nonce_le), crates/flock-core/src/challenger.rs:1100-1140).
#pragma once
#include <cstdint>

namespace flock {
namespace gpu {

__constant__ static uint32_t SHA_K[64] = {
    0x428a2f98, 0x71374491, 0xb5c0fbcf, 0xe9b5dba5, 0x3956c25b, 0x59f111f1, 0x923f82a4, 0xab1c5ed5,
    0xd807aa98, 0x12835b01, 0x243185be, 0x550c7dc3, 0x72be5d74, 0x80deb1fe, 0x9bdc06a7, 0xc19bf174,
    0xe49b69c1, 0xefbe4786, 0x0fc19dc6, 0x240ca1cc, 0x2de92c6f, 0x4a7484aa, 0x5cb0a9dc, 0x76f988da,
    0x983e5152, 0xa831c66d, 0xb00327c8, 0xbf597fc7, 0xc6e00bf3, 0xd5a79147, 0x06ca6351, 0x14292967,
    0x27b70a85, 0x2e1b2138, 0x4d2c6dfc, 0x53380d13, 0x650a7354, 0x766a0abb, 0x81c2c92e, 0x92722c85,
    0xa2bfe8a1, 0xa81a664b, 0xc24b8b70, 0xc76c51a3, 0xd192e819, 0xd6990624, 0xf40e3585, 0x106aa070,
    0x19a4c116, 0x1e376c08, 0x2748774c, 0x34b0bcb5, 0x391c0cb3, 0x4ed8aa4a, 0x5b9cca4f, 0x682e6ff3,
    0x748f82ee, 0x78a5636f, 0x84c87814, 0x8cc70208, 0x90befffa, 0xa4506ceb, 0xbef9a3f7, 0xc67178f2};

// __host__ as well: the host-side tests of the device transcript run the same code.
__host__ __device__ __forceinline__ uint32_t rotr(uint32_t x, int n) {
#ifdef __CUDA_ARCH__
  return __funnelshift_r(x, x, n);
#else
  return (x >> n) | (x << (32 - n));
#endif
}
__host__ __device__ __forceinline__ uint32_t bswap32(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __byte_perm(x, 0, 0x0123);
#else
  return (x >> 24) | ((x >> 8) & 0xFF00u) | ((x << 8) & 0xFF0000u) | (x << 24);
#endif
}
__host__ __device__ __forceinline__ uint32_t sha_k(int i) {
#ifdef __CUDA_ARCH__
  return SHA_K[i];
#else
  static const uint32_t K[64] = {
      0x428a2f98, 0x71374491, 0xb5c0fbcf, 0xe9b5dba5, 0x3956c25b, 0x59f111f1, 0x923f82a4, 0xab1c5ed5,
      0xd807aa98, 0x12835b01, 0x243185be, 0x550c7dc3, 0x72be5d74, 0x80deb1fe, 0x9bdc06a7, 0xc19bf174,
      0xe49b69c1, 0xefbe4786, 0x0fc19dc6, 0x240ca1cc, 0x2de92c6f, 0x4a7484aa, 0x5cb0a9dc, 0x76f988da,
      0x983e5152, 0xa831c66d, 0xb00327c8, 0xbf597fc7, 0xc6e00bf3, 0xd5a79147, 0x06ca6351, 0x14292967,
      0x27b70a85, 0x2e1b2138, 0x4d2c6dfc, 0x53380d13, 0x650a7354, 0x766a0abb, 0x81c2c92e, 0x92722c85,
      0xa2bfe8a1, 0xa81a664b, 0xc24b8b70, 0xc76c51a3, 0xd192e819, 0xd6990624, 0xf40e3585, 0x106aa070,
      0x19a4c116, 0x1e376c08, 0x2748774c, 0x34b0bcb5, 0x391c0cb3, 0x4ed8aa4a, 0x5b9cca4f, 0x682e6ff3,
      0x748f82ee, 0x78a5636f, 0x84c87814, 0x8cc70208, 0x90befffa, 0xa4506ceb, 0xbef9a3f7, 0xc67178f2};
  return K[i];
#endif
}

// MULADD: x + y on the multiply pipe (x * 1 + y with the one in constant memory, which keeps it a
// multiply-add). The compression's rotations, choices and adds otherwise all run on the logic
// pipe, which bounded the large Merkle levels (94 % busy, the multiply pipe 10 %): with every add
// moved over, the leaves of 2^20 rows of 42 words take 0.71 ms instead of 0.82 (half of the adds:
// 0.80). Two-operand adds make longer chains than three-operand ones, so where a launch is bound
// by one compression's latency the plain adds are faster (Merkle stages of BLAKE3 2^12 0.158
// against 0.171 ms).
__constant__ static uint32_t SHA_ONE = 1;
template <bool MULADD>
__host__ __device__ __forceinline__ uint32_t sha_add(uint32_t x, uint32_t y) {
#ifdef __CUDA_ARCH__
  if (MULADD) {
    uint32_t r;
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(x), "r"(SHA_ONE), "r"(y));
    return r;
  }
#endif
  return x + y;
}

// One compression; w[0..16] are the block's big-endian words.
template <bool MULADD = false>
__host__ __device__ __forceinline__ void sha256_compress(uint32_t st[8], uint32_t w[16]) {
  uint32_t a = st[0], b = st[1], c = st[2], d = st[3], e = st[4], f = st[5], g = st[6], h = st[7];
#pragma unroll
  for (int i = 0; i < 64; ++i) {
    uint32_t wi;
    if (i < 16) {
      wi = w[i];
    } else {
      uint32_t w15 = w[(i + 1) & 15], w2 = w[(i + 14) & 15];
      uint32_t s0 = rotr(w15, 7) ^ rotr(w15, 18) ^ (w15 >> 3);
      uint32_t s1 = rotr(w2, 17) ^ rotr(w2, 19) ^ (w2 >> 10);
      wi = MULADD ? sha_add<MULADD>(sha_add<MULADD>(sha_add<MULADD>(w[i & 15], w[(i + 9) & 15]), s0), s1)
                  : w[i & 15] + s0 + w[(i + 9) & 15] + s1;
      w[i & 15] = wi;
    }
    uint32_t S1 = rotr(e, 6) ^ rotr(e, 11) ^ rotr(e, 25);
    uint32_t ch = (e & f) ^ (~e & g);
    uint32_t t1 = MULADD ? sha_add<MULADD>(sha_add<MULADD>(sha_add<MULADD>(sha_add<MULADD>(h, sha_k(i)), wi), ch), S1)
                         : h + S1 + ch + sha_k(i) + wi;
    uint32_t S0 = rotr(a, 2) ^ rotr(a, 13) ^ rotr(a, 22);
    uint32_t mj = (a & b) ^ (a & c) ^ (b & c);
    h = g; g = f; f = e; e = sha_add<MULADD>(d, t1); d = c; c = b; b = a; a = MULADD ? sha_add<MULADD>(sha_add<MULADD>(S0, mj), t1) : t1 + S0 + mj;
  }
  st[0] += a; st[1] += b; st[2] += c; st[3] += d; st[4] += e; st[5] += f; st[6] += g; st[7] += h;
}

__host__ __device__ __forceinline__ void sha256_init(uint32_t st[8]) {
  st[0] = 0x6a09e667; st[1] = 0xbb67ae85; st[2] = 0x3c6ef372; st[3] = 0xa54ff53a;
  st[4] = 0x510e527f; st[5] = 0x9b05688c; st[6] = 0x1f83d9ab; st[7] = 0x5be0cd19;
}

// SHA-256 of `nwords` little-endian u32 words (byte length 4 * nwords, a multiple of 16).
// The message is read through `load(i)` returning the i-th LE word.
template <bool MULADD = false, class Load>
__device__ __forceinline__ void sha256_words(Load load, uint32_t nwords, uint32_t out[8]) {
  uint32_t st[8];
  sha256_init(st);
  uint32_t w[16];
  uint32_t full = nwords / 16;
  for (uint32_t blk = 0; blk < full; ++blk) {
#pragma unroll
    for (int i = 0; i < 16; ++i) w[i] = bswap32(load(blk * 16 + i));
    sha256_compress<MULADD>(st, w);
  }
  uint32_t rem = nwords - full * 16;  // 0, 4, 8 or 12 words
  uint64_t bits = (uint64_t)nwords * 32;
#pragma unroll
  for (int i = 0; i < 16; ++i) w[i] = 0;
  for (uint32_t i = 0; i < rem; ++i) w[i] = bswap32(load(full * 16 + i));
  w[rem] = 0x80000000u;
  if (rem >= 14) {
    sha256_compress<MULADD>(st, w);
#pragma unroll
    for (int i = 0; i < 16; ++i) w[i] = 0;
  }
  w[14] = (uint32_t)(bits >> 32);
  w[15] = (uint32_t)bits;
  sha256_compress<MULADD>(st, w);
#pragma unroll
  for (int i = 0; i < 8; ++i) out[i] = bswap32(st[i]);  // digest bytes as LE words
}

}  // namespace gpu
}  // namespace flock
