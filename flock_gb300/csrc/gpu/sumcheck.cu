// Sumcheck-side kernels of prove_fast: the zerocheck round 1 on the skip domain and
// its folds, the lincheck column folds / row fold / product sumcheck, the merged-open
// weight build and folds, and the Ligerito F256 ladder (basis tables, folds, messages,
// code switch, induced basis).
//
// Reductions: every message kernel writes per-block XOR partials to `part`
// (part[block * width + j]); the last block to arrive XORs them into `width` values
// and publishes these to mapped memory.
// Eq tables over many variables are never materialised: eq(i) = lo[i & (2^lo_bits - 1)]
// * hi[i >> lo_bits], and kernels that sum eq-weighted terms walk chunks of 2^lo_bits
// consecutive indices, summing lo-weighted terms and multiplying by hi once per chunk.
#include "kernels.h"
#include "reduce.cuh"
#include "wintable.cuh"
#include <atomic>
#include <mutex>
#include <set>
#include <tuple>
#include <type_traits>

namespace flock {
namespace gpu {

// ------------------------------------------------------------------ generic pieces
// Both tables of an eq split in one launch: lo = eq(p[0 .. lo_bits)) and
// hi = scale * eq(p[lo_bits .. lo_bits + hi_bits)); entry e < 2^lo_bits is a lo entry.
__global__ void __launch_bounds__(EQ_THREADS)
eq_split_kernel(const F128d* __restrict__ p, uint32_t lo_bits, uint32_t hi_bits, F128d scale, F128d* __restrict__ lo,
                F128d* __restrict__ hi) {
  __shared__ F128d sub[2][EQ_MAX_GROUPS][16];
  eq_sub_tables(p, lo_bits, sub[0]);
  eq_sub_tables(p + lo_bits, hi_bits, sub[1]);
  __syncthreads();
  const uint64_t n_lo = 1ull << lo_bits, n = n_lo + (1ull << hi_bits);
  const bool scaled = scale.lo != 1 || scale.hi != 0;
  for (uint64_t e = (uint64_t)blockIdx.x * EQ_THREADS + threadIdx.x; e < n; e += (uint64_t)gridDim.x * EQ_THREADS) {
    if (e < n_lo) {
      lo[e] = eq_from_sub(sub[0], lo_bits, e);
    } else {
      const F128d v = eq_from_sub(sub[1], hi_bits, e - n_lo);
      hi[e - n_lo] = scaled ? mul_call(scale, v) : v;
    }
  }
}
void launch_eq_split(const F128d* d_point, uint32_t lo_bits, uint32_t hi_bits, F128d scale, F128d* lo, F128d* hi,
                     cudaStream_t s) {
  const uint64_t len = (1ull << lo_bits) + (1ull << hi_bits);
  const uint32_t blocks = (uint32_t)std::min<uint64_t>((len + EQ_THREADS - 1) / EQ_THREADS, (uint64_t)sm_count() * 8);
  eq_split_kernel<<<blocks, EQ_THREADS, 0, s>>>(d_point, lo_bits, hi_bits, scale, lo, hi);
  LAUNCH_OK();
}

// XOR of the rows of two partial arrays (na rows of width wa, nb of width wb), published side by
// side; one block a value (46 values of 360 rows by one block, which this replaced: 30 us).
__global__ void __launch_bounds__(128)
reduce_pair_kernel(const F128d* __restrict__ pa, uint32_t na, uint32_t wa, const F128d* __restrict__ pb, uint32_t nb,
                   uint32_t wb, FusedPublish pub) {
  __shared__ F128d sh[32];
  const bool second = blockIdx.x >= wa;
  const F128d* p = second ? pb + (blockIdx.x - wa) : pa + blockIdx.x;
  const uint32_t n = second ? nb : na, w = second ? wb : wa;
  F128d acc = f128_zero();
  for (uint32_t b = threadIdx.x; b < n; b += blockDim.x) acc += p[(uint64_t)b * w];
  acc = block_xor(acc, sh);
  if (threadIdx.x == 0) pub.out[blockIdx.x] = acc;
  publish_data(pub);
}
void launch_reduce_pair(const F128d* pa, uint32_t na, uint32_t wa, const F128d* pb, uint32_t nb, uint32_t wb,
                        cudaStream_t s, FusedPublish pub) {
  reduce_pair_kernel<<<wa + wb, 128, 0, s>>>(pa, na, wa, pb, nb, wb, pub);
  LAUNCH_OK();
}

static std::atomic<uint64_t> g_launches{0};
uint64_t launch_count() { return g_launches.load(std::memory_order_relaxed); }
void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

static int current_device() {
  int dev = 0;
  CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= MAX_DEVICES) throw std::runtime_error("device index out of range");
  return dev;
}
int sm_count() {
  static std::atomic<int> cache[MAX_DEVICES];
  const int dev = current_device();
  int n = cache[dev].load(std::memory_order_relaxed);
  if (!n) {
    CUDA_OK(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    cache[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}
void set_dynamic_smem(const void* kernel, int bytes) {
  static std::mutex mu;
  static std::set<std::tuple<const void*, int, int>> done;
  const auto key = std::make_tuple(kernel, current_device(), bytes);
  std::lock_guard<std::mutex> g(mu);
  if (done.count(key)) return;
  CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  done.insert(key);
}

// ------------------------------------------------------------------ bit sums
// U[col][t] = sum_row eq(row) * bit_t(z[col * col_stride + row * row_stride]) over the 128 bits of
// each word: the s_hat_v_c sums of the zerocheck (rows = xo, columns = the 64 words of an xo),
// the lincheck's row fold (rows = instances, columns = chunk columns) and Ligerito's lane dots
// (rows of a lane; sum_t x^t U[lane][t] is the field dot product, so it needs no product a word).
// No multiply: 32 rows at a time, a warp transposes a column's 32 words (lane c then holds, per
// 32-bit limb, bit c of all 32 rows) and looks up the subset sums of the rows' eq weights, in
// windows of 7, 7, 6, 6 and 6 rows. The tables depend on the rows alone and serve every column of
// the block, so they are stored eight times, once per bank group (wintable.cuh): no lookup
// conflicts. Per word 20 lookups and 20 shuffles of a warp over 32 words: 3.1 cycles of the
// shared-memory pipe, plus the build (448 stores a tile) shared by up to 64 columns. Two table
// buffers, one barrier a tile. eq(row) = eq_lo[row mod 2^lo_bits] eq_hi[row >> lo_bits], 512 rows'
// products at a time. The forms it replaced read four- and eight-row tables with
// conflicts or took field products: Keccak-f 2^18 (87 M words) s_hat_v_c 4.7 -> 1.7 ms, lincheck
// row fold 3.9 -> 1.4, lane dots 1.6 -> 1.5; SHA-256 2^16 0.69 -> 0.34, 0.55 -> 0.19, 0.51 -> 0.27.
enum BitSumOut : int {
  BITS_RAW,      // part[(col * splits + split) * 128 + t] = U
  BITS_COLUMNS,  // part[(split * groups + group) * 128 + t] = sum over the group's columns of weight[col] U
  BITS_DOT,      // part[split * n_cols + col] = sum_t x^t U
  BITS_POINTS,   // the words of zc_round1_bits: part[(split * groups + group) * 64 + i] = the group's share of
                 // sum_{M, bit} weight[8 M + bit] U at point i
};
constexpr uint32_t BITS_EQ_ROWS = 512;
constexpr uint32_t BITS_TABLE_BYTES = (2 * 128 + 3 * 64) * 128;
// Warp-wide 32 x 32 bit transpose: lane r holds word x_r; afterwards lane c holds the word
// whose bit r is bit c of x_r (five exchange stages of halving block size).
__device__ __forceinline__ uint32_t warp_transpose32(uint32_t x) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t masks[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const uint32_t j = 16u >> s, m = masks[s];
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, j);
    x = (lane & j) ? ((x & ~m) | ((y & ~m) >> j)) : ((x & m) | ((y & m) << j));
  }
  return x;
}

__device__ __forceinline__ void build_bit_tables(const F128d* e, char* T) {
  // a team of eight threads (one per copy) walks eight entries: 16 teams for each seven-row
  // window, 8 for each six-row one
  const uint32_t team = threadIdx.x >> 3, r = threadIdx.x & 7;
  if (team >= 56) return;
  const uint32_t win = team < 32 ? team >> 4 : 2 + ((team - 32) >> 3);
  const uint32_t hi = team < 32 ? team & 15 : team & 7;                    // the entry's bits from 3 on
  const uint32_t row0 = win < 2 ? 7 * win : 14 + 6 * (win - 2);
  const uint32_t ent0 = (win < 2 ? 128 * win : 256 + 64 * (win - 2)) + 8 * hi;
  F128d acc = f128_zero();
#pragma unroll
  for (uint32_t b = 0; b < 4; ++b) {
    const uint64_t m = 0ull - (uint64_t)((hi >> b) & 1);
    const F128d w = e[min(row0 + 3 + b, 31u)];  // b = 3 is never set in a six-row window
    acc.lo ^= w.lo & m;
    acc.hi ^= w.hi & m;
  }
  const F128d e0 = e[row0], e1 = e[row0 + 1], e2 = e[row0 + 2];
  char* o = T + ent0 * 128 + r * 16;
  auto put = [&](uint32_t v) { *reinterpret_cast<F128d*>(o + v * 128) = acc; };
  put(0);
  acc += e0; put(1);
  acc += e1; put(3);
  acc += e0; put(2);
  acc += e2; put(6);
  acc += e0; put(7);
  acc += e1; put(5);
  acc += e0; put(4);
}
template <int CPW, int OUT>
__global__ void __launch_bounds__(BITS_THREADS, 1)
bit_sums_kernel(const F128d* __restrict__ z, uint64_t col_stride, uint64_t row_stride, uint32_t n_cols, uint64_t n_rows,
                uint64_t rows_per_split, const F128d* __restrict__ eq_lo, uint32_t lo_bits,
                const F128d* __restrict__ eq_hi, const F128d* __restrict__ weight, F128d* __restrict__ part) {
  extern __shared__ __align__(16) char bt[];  // two tables
  __shared__ F128d eq[2][BITS_EQ_ROWS];       // this stage's row weights and the next one's
  const uint32_t warp = threadIdx.x >> 5, t = threadIdx.x & 31, lane16 = win_lane();
  const uint32_t col0 = (blockIdx.x * BITS_WARPS + warp) * CPW;
  const uint64_t row_begin = (uint64_t)blockIdx.y * rows_per_split;
  const uint64_t row_end = min(n_rows, row_begin + rows_per_split);
  auto stage_eq = [&](uint64_t row, uint32_t buf) {
    F128d v = f128_zero();  // rows past the end weigh nothing
    if (row + threadIdx.x < row_end) {
      const uint64_t x = row + threadIdx.x;
      v = mul_call(eq_lo[x & ((1ull << lo_bits) - 1)], eq_hi[x >> lo_bits]);
    }
    eq[buf][threadIdx.x] = v;
  };
  F128d U[CPW][4];
#pragma unroll
  for (int c = 0; c < CPW; ++c)
#pragma unroll
    for (int q = 0; q < 4; ++q) U[c][q] = f128_zero();
  if (row_begin < row_end) {
    const uint32_t tiles = (uint32_t)((row_end - row_begin + 31) / 32);
    constexpr uint32_t STAGE = BITS_EQ_ROWS / 32;  // tiles per eq stage
    stage_eq(row_begin, 0);
    __syncthreads();
    build_bit_tables(eq[0], bt);
    for (uint32_t i = 0; i < tiles; ++i) {
      const uint64_t row = row_begin + (uint64_t)i * 32 + t;
      uint4 x[CPW];
#pragma unroll
      for (int c = 0; c < CPW; ++c)
        x[c] = col0 + c < n_cols && row < row_end
                   ? *reinterpret_cast<const uint4*>(z + (col0 + c) * col_stride + row * row_stride)
                   : make_uint4(0, 0, 0, 0);
      // the next stage's weights, written a tile before the first table that reads them is built
      if (i % STAGE == STAGE - 2) stage_eq(row_begin + (uint64_t)(i / STAGE + 1) * BITS_EQ_ROWS, (i / STAGE + 1) & 1);
      __syncthreads();  // this tile's table is complete, the other buffer no longer read
      if (i + 1 < tiles)
        build_bit_tables(eq[((i + 1) / STAGE) & 1] + 32 * ((i + 1) % STAGE), bt + ((i + 1) & 1) * BITS_TABLE_BYTES);
      const char* T = bt + (i & 1) * BITS_TABLE_BYTES;
      if (col0 < n_cols) {  // warp-uniform
#pragma unroll
        for (int c = 0; c < CPW; ++c) {
          const uint32_t w[4] = {x[c].x, x[c].y, x[c].z, x[c].w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint32_t y = warp_transpose32(w[q]);
            const uint32_t o[5] = {((y << 7) & (127u << 7)) | lane16, (y & (127u << 7)) | lane16,
                                   ((y >> 7) & (63u << 7)) | lane16, ((y >> 13) & (63u << 7)) | lane16,
                                   ((y >> 19) & (63u << 7)) | lane16};
            U[c][q] += *reinterpret_cast<const F128d*>(T + o[0]);
            U[c][q] += *reinterpret_cast<const F128d*>(T + 128 * 128 + o[1]);
            U[c][q] += *reinterpret_cast<const F128d*>(T + 256 * 128 + o[2]);
            U[c][q] += *reinterpret_cast<const F128d*>(T + 320 * 128 + o[3]);
            U[c][q] += *reinterpret_cast<const F128d*>(T + 384 * 128 + o[4]);
          }
        }
      }
    }
  }
  if (OUT == BITS_RAW) {
#pragma unroll
    for (int c = 0; c < CPW; ++c)
      if (col0 + c < n_cols)
#pragma unroll
        for (int q = 0; q < 4; ++q) part[((uint64_t)(col0 + c) * gridDim.y + blockIdx.y) * 128 + 32 * q + t] = U[c][q];
  } else if (OUT == BITS_DOT) {
#pragma unroll
    for (int c = 0; c < CPW; ++c) {
      F128d v = f128_zero();
#pragma unroll
      for (int q = 0; q < 4; ++q) v += mul_by_power(U[c][q], 32 * q + t);
      v = warp_xor(v);
      if (t == 0 && col0 + c < n_cols) part[(uint64_t)blockIdx.y * n_cols + col0 + c] = v;
    }
  } else if (OUT == BITS_POINTS) {
    F128d* red = reinterpret_cast<F128d*>(bt);  // [column of the group][16 points]
    __syncthreads();
#pragma unroll
    for (int c = 0; c < CPW; ++c) {
      F128d v = f128_zero();
      const uint32_t w = col0 + c, m0 = 2 * (w >> 3), h = w & 1;  // w = 8 (M / 2) + 2 q + h
#pragma unroll
      for (int l = 0; l < 4; ++l) v += mul_call(weight[8 * ((m0 + (t >> 4)) & 15) + 4 * h + l], U[c][l]);
      v.lo ^= __shfl_xor_sync(0xffffffffu, v.lo, 16);
      v.hi ^= __shfl_xor_sync(0xffffffffu, v.hi, 16);
      if (t < 16) red[(warp * CPW + c) * 16 + t] = v;
    }
    __syncthreads();
    if (threadIdx.x < 64) {
      const uint32_t q = threadIdx.x >> 4;
      F128d acc = f128_zero();
      for (uint32_t c = 0; c < BITS_WARPS * CPW; ++c) {
        const uint32_t w = blockIdx.x * BITS_WARPS * CPW + c;
        if (w < n_cols && ((w >> 1) & 3) == q) acc += red[c * 16 + (threadIdx.x & 15)];
      }
      part[((uint64_t)blockIdx.y * gridDim.x + blockIdx.x) * 64 + threadIdx.x] = acc;
    }
  } else {
    F128d v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = f128_zero();
#pragma unroll
    for (int c = 0; c < CPW; ++c)
      if (col0 + c < n_cols)
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] += mul_call(weight[col0 + c], U[c][q]);
    F128d* red = reinterpret_cast<F128d*>(bt);  // [warp][128]
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) red[warp * 128 + 32 * q + t] = v[q];
    __syncthreads();
    if (threadIdx.x < 128) {
      F128d a = f128_zero();
      for (uint32_t w = 0; w < BITS_WARPS; ++w) a += red[w * 128 + threadIdx.x];
      part[((uint64_t)blockIdx.y * gridDim.x + blockIdx.x) * 128 + threadIdx.x] = a;
    }
  }
}
template <int CPW, int OUT>
static void bit_sums_cpw(const BitSumPlan& p, const F128d* z, uint64_t col_stride, uint64_t row_stride, uint32_t n_cols,
                         uint64_t n_rows, const F128d* eq_lo, uint32_t lo_bits, const F128d* eq_hi, const F128d* weight,
                         F128d* part, cudaStream_t s) {
  const int smem = 2 * (int)BITS_TABLE_BYTES;
  set_dynamic_smem((const void*)bit_sums_kernel<CPW, OUT>, smem);
  bit_sums_kernel<CPW, OUT><<<dim3(p.groups, p.splits), BITS_THREADS, smem, s>>>(
      z, col_stride, row_stride, n_cols, n_rows, p.rows_per_split, eq_lo, lo_bits, eq_hi, weight, part);
  LAUNCH_OK();
}
template <int OUT>
static void bit_sums(const BitSumPlan& p, const F128d* z, uint64_t col_stride, uint64_t row_stride, uint32_t n_cols,
                     uint64_t n_rows, const F128d* eq_lo, uint32_t lo_bits, const F128d* eq_hi, const F128d* weight,
                     F128d* part, cudaStream_t s) {
  switch (p.cpw) {
    case 1: return bit_sums_cpw<1, OUT>(p, z, col_stride, row_stride, n_cols, n_rows, eq_lo, lo_bits, eq_hi, weight, part, s);
    case 2: return bit_sums_cpw<2, OUT>(p, z, col_stride, row_stride, n_cols, n_rows, eq_lo, lo_bits, eq_hi, weight, part, s);
    case 3: return bit_sums_cpw<3, OUT>(p, z, col_stride, row_stride, n_cols, n_rows, eq_lo, lo_bits, eq_hi, weight, part, s);
    default: return bit_sums_cpw<4, OUT>(p, z, col_stride, row_stride, n_cols, n_rows, eq_lo, lo_bits, eq_hi, weight, part, s);
  }
}

// ------------------------------------------------------------------ zerocheck round 1
// With the fixed challenges r[6..13) the row eq factorises. For a row x (m - 6 bits)
// = (K: 3 bits, M: 4 bits, xo):
//   eq(r[6..m], x) = phi8(e_K) * D * x^M * eq(r[13..m], xo),
// e_K = prod_j (K_j ? c_j : 1 + c_j) over the three GF(2^8) constants c_j (phi8 is a
// ring embedding), and D = prod_i (1 + g_i)^-1 over the medium constants g_i = x^(2^i)
// (the bit-1 factor g/(1+g) and the bit-0 factor 1/(1+g)). Hence per Lambda point i
//   P_ab(i) = D * sum_xo eq_o(xo) * sum_M x^M * phi8( sum_K e_K * ext(a_x)(i) * ext(b_x)(i) )
// where the inner sums are GF(2^8) byte arithmetic and each xo costs one F128 multiply
// per output. The same factorisation over words w = (K2: 2 bits, M, xo) with e2 over
// r[7], r[8] gives s_hat_v_c[t] from bit t of z_w. P_c needs no pass of its own: it is
// linear in the z bits and the host derives it from s_hat_v_c. D is applied by the host.
// For P_ab the inner sums g_M(i) = sum_K e_K ext(a_x)(i) ext(b_x)(i) are formed as bits (below), and
// since phi8 is additive the outer sums are bit sums:
//   P_ab(i) = D * sum_{M, bit} x^M phi8(2^bit) * sum_xo eq_o(xo) * bit(g_M(i) of xo).
constexpr uint32_t ZC_WINDOWS = 9;                           // of a 64-bit row: eight of 7 bits, one of 8
constexpr uint32_t ZC_EXT_ENTRIES = 8 * 128 + 256;
constexpr uint32_t ZC_EXT_BYTES = ZC_EXT_ENTRIES * 128;      // two 64-byte copies an entry
struct ZcConsts {
  uint8_t ext[ZC_EXT_ENTRIES][64];  // extension of the window's bits, see upload_zc_consts
  F128d wconst[64];                 // word weights within an xo: x^M * phi8(e2[K2]) for word 4M + K2
  F128d pconst[128];                // x^M * phi8(2^bit) at 8 M + bit
};

__host__ __device__ constexpr uint32_t gf8_const_mul(uint32_t a, uint32_t b) {
  uint32_t r = 0;
  for (int k = 0; k < 8; ++k) {
    if ((b >> k) & 1) r ^= a;
    a = (a << 1) ^ ((a & 0x80) ? 0x11Bu : 0u);
  }
  return r & 0xFF;
}
// e_K over the three small constants of the zerocheck.
__host__ __device__ constexpr uint32_t zc_e(int K) {
  return gf8_const_mul(gf8_const_mul((K & 1) ? 0xF7u : 0xF6u, (K & 2) ? 0x53u : 0x52u), (K & 4) ? 0xB5u : 0xB4u);
}
// Where window k of a row starts.
__host__ __device__ constexpr uint32_t zc_window_bit(uint32_t k) { return 7 * k; }

// g += e_K * a * b for 32 pairs of GF(2^8) elements given as eight bit planes each: the fifteen
// planes of the carry-less products, then the map c -> e_K c mod (x^8 + x^4 + x^3 + x + 1), whose
// matrix is constant.
template <int K>
__device__ __forceinline__ void gf8_planes_mac(const uint32_t a[8], const uint32_t b[8], uint32_t g[8]) {
  uint32_t c[15];
#pragma unroll
  for (int k = 0; k < 15; ++k) {
    c[k] = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (k - i >= 0 && k - i < 8) c[k] ^= a[i] & b[k - i];
  }
#pragma unroll
  for (int k = 14; k >= 8; --k) {
    c[k - 4] ^= c[k];
    c[k - 5] ^= c[k];
    c[k - 7] ^= c[k];
    c[k - 8] ^= c[k];
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t col = gf8_const_mul(zc_e(K), 1u << j);  // e_K x^j
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if ((col >> i) & 1) g[i] ^= c[j];
  }
}

// g_M of every live xo as bits. A team of four lanes takes the row pairs (8M + K, 8(M+1) + K) of one
// even M, lane q the points 16q .. 16q + 15: per row nine lookups of 16 bytes in the extension
// tables, stored so that register r of an entry holds bit planes 2r (low half) and 2r + 1 of the
// lane's 16 points; one byte permute per plane pair then sets the two rows side by side, and the
// GF(2^8) products run on planes of 32 elements. A warp is one xo (eight teams, its 2 KB of a and
// b read once); eight consecutive lanes are two teams, which read different copies of the 64-byte
// entries, so no lookup conflicts. Per xo 1152 cycles of the shared-memory pipe (9 a row) and
// about 1100 of the logic pipe. The form it replaced took 3160 (byte tables read with conflicts,
// products from a 64 KB table and byte by byte, one F128 product an xo and point, a block per 32
// xo): the whole round, with both bit sums, Keccak-f 2^18 15.4 -> 8.9 ms, SHA-256 2^16 2.41 -> 1.41,
// BLAKE3 2^8 105 -> 42 us. Output word 8 (M / 2) + 2 q + h of the xo: limb l is plane 4 h + l, bits 0-15 the points
// at M, bits 16-31 those at M + 1.
constexpr uint32_t ZC_R1_THREADS = 512;
__global__ void __launch_bounds__(ZC_R1_THREADS, 1)
zc_round1_bits_kernel(const F128d* __restrict__ a, const F128d* __restrict__ b, uint64_t n_xo,
                      const ZcConsts* __restrict__ gconst, uint4* __restrict__ g_out) {
  extern __shared__ __align__(16) char ext[];  // ZC_EXT_BYTES
  for (uint32_t i = threadIdx.x; i < ZC_EXT_ENTRIES * 4; i += ZC_R1_THREADS) {
    const uint4 v = reinterpret_cast<const uint4*>(gconst->ext)[i];
    uint4* o = reinterpret_cast<uint4*>(ext + (i >> 2) * 128) + (i & 3);
    o[0] = v;
    o[4] = v;
  }
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31, mp = lane >> 2;
  const uint32_t off = (mp & 1) * 64 + (lane & 3) * 16;  // this team's copy, this lane's points
  auto extend = [&](uint32_t lo, uint32_t hi) {
    constexpr uint32_t M7 = 127u << 7;
    const uint32_t o[ZC_WINDOWS] = {(lo << 7) & M7, lo & M7, (lo >> 7) & M7, (lo >> 14) & M7,
                                    __funnelshift_r(lo, hi, 21) & M7, (hi << 4) & M7, (hi >> 3) & M7, (hi >> 10) & M7,
                                    (hi >> 17) & (255u << 7)};
    uint4 r = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (uint32_t k = 0; k < ZC_WINDOWS; ++k) {
      const uint4 t = *reinterpret_cast<const uint4*>(ext + k * 128 * 128 + (o[k] | off));
      r.x ^= t.x;
      r.y ^= t.y;
      r.z ^= t.z;
      r.w ^= t.w;
    }
    return r;
  };
  auto planes = [](uint4 x, uint4 y, uint32_t o[8]) {  // rows of M and M + 1 side by side
    o[0] = __byte_perm(x.x, y.x, 0x5410); o[1] = __byte_perm(x.x, y.x, 0x7632);
    o[2] = __byte_perm(x.y, y.y, 0x5410); o[3] = __byte_perm(x.y, y.y, 0x7632);
    o[4] = __byte_perm(x.z, y.z, 0x5410); o[5] = __byte_perm(x.z, y.z, 0x7632);
    o[6] = __byte_perm(x.w, y.w, 0x5410); o[7] = __byte_perm(x.w, y.w, 0x7632);
  };
  for (uint64_t xo = (uint64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x; xo < n_xo;
       xo += (uint64_t)gridDim.x * (ZC_R1_THREADS / 32)) {
    const uint4* wa = reinterpret_cast<const uint4*>(a + xo * 64) + 8 * mp;  // words of M, then of M + 1
    const uint4* wb = reinterpret_cast<const uint4*>(b + xo * 64) + 8 * mp;
    uint32_t g[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) g[i] = 0;
    auto rows = [&](auto kk) {  // the word's two rows K = 2 kk and 2 kk + 1
      constexpr int k2 = decltype(kk)::value;
      const uint4 A0 = wa[k2], A1 = wa[4 + k2], B0 = wb[k2], B1 = wb[4 + k2];
      uint32_t pa[8], pb[8];
      planes(extend(A0.x, A0.y), extend(A1.x, A1.y), pa);
      planes(extend(B0.x, B0.y), extend(B1.x, B1.y), pb);
      gf8_planes_mac<2 * k2>(pa, pb, g);
      planes(extend(A0.z, A0.w), extend(A1.z, A1.w), pa);
      planes(extend(B0.z, B0.w), extend(B1.z, B1.w), pb);
      gf8_planes_mac<2 * k2 + 1>(pa, pb, g);
    };
    rows(std::integral_constant<int, 0>());
    rows(std::integral_constant<int, 1>());
    rows(std::integral_constant<int, 2>());
    rows(std::integral_constant<int, 3>());
    uint4* o = g_out + xo * 64 + 8 * mp + 2 * (lane & 3);
    o[0] = make_uint4(g[0], g[1], g[2], g[3]);
    o[1] = make_uint4(g[4], g[5], g[6], g[7]);
  }
}

static ZcConsts* g_zc_consts_dev[MAX_DEVICES] = {};  // written under the caller's lock, before any prover launches
static ZcConsts* zc_consts() { return g_zc_consts_dev[current_device()]; }
// unit[64 s + i]: the extension of row bit s at Lambda point i.
void upload_zc_consts(const uint8_t* unit, const F128d* wconst, const F128d* pconst) {
  const int dev = current_device();
  if (g_zc_consts_dev[dev]) return;
  ZcConsts* h = new ZcConsts();
  for (uint32_t e = 0; e < ZC_EXT_ENTRIES; ++e) {
    const uint32_t k = std::min(e >> 7, ZC_WINDOWS - 1), v = e - (k << 7);
    for (uint32_t i = 0; i < 64; ++i) {
      uint8_t x = 0;
      for (uint32_t bit = 0; bit < 8; ++bit)
        if ((v >> bit) & 1) x ^= unit[64 * (zc_window_bit(k) + bit) + i];
      // plane p of points 16q .. 16q + 15: half p & 1 of 32-bit word 4 q + p / 2
      for (uint32_t p = 0; p < 8; ++p)
        if ((x >> p) & 1) {
          const uint32_t pos = (i & 15) + 16 * (p & 1);
          h->ext[e][16 * (i >> 4) + 4 * (p >> 1) + (pos >> 3)] |= (uint8_t)(1u << (pos & 7));
        }
    }
  }
  memcpy(h->wconst, wconst, sizeof(h->wconst));
  memcpy(h->pconst, pconst, sizeof(h->pconst));
  ZcConsts* d = nullptr;
  CUDA_OK(cudaMalloc(&d, sizeof(ZcConsts)));
  CUDA_OK(cudaMemcpy(d, h, sizeof(ZcConsts), cudaMemcpyHostToDevice));
  CUDA_OK(cudaDeviceSynchronize());  // complete before any kernel of a non-blocking stream reads it
  delete h;
  g_zc_consts_dev[dev] = d;
}

void launch_zc_round1(const F128d* a, const F128d* b, const F128d* z, uint32_t m, uint64_t live_words,
                      const F128d* eq_lo, uint32_t lo_bits, const F128d* eq_hi, F128d* g, F128d* part_ab,
                      F128d* part_svc, uint64_t part_room, uint32_t* nrows, cudaStream_t s) {
  const ZcConsts* consts = zc_consts();
  if (!consts) throw std::runtime_error("zerocheck constants not uploaded");
  // xo past the live words hold zero rows of z, a and b and add nothing to any sum
  const uint64_t xo_live = std::min<uint64_t>(1ull << (m - 13), (live_words + 63) / 64);
  const BitSumPlan p = bit_sum_plan(64, xo_live, BITS_MAX_SPLITS, (uint64_t)sm_count());
  if (uint64_t(p.groups) * p.splits * 128 > part_room) throw std::runtime_error("round-1 partials exceed the partials buffer");
  set_dynamic_smem((const void*)zc_round1_bits_kernel, (int)ZC_EXT_BYTES);
  // one block per SM; xo are dealt to the blocks first, then to their warps
  const uint32_t blocks = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(xo_live, (uint64_t)sm_count()));
  zc_round1_bits_kernel<<<blocks, ZC_R1_THREADS, ZC_EXT_BYTES, s>>>(a, b, xo_live, consts, reinterpret_cast<uint4*>(g));
  LAUNCH_OK();
  // both outer sums: 64 words an xo, rows = xo
  bit_sums<BITS_POINTS>(p, g, 1, 64, 64, xo_live, eq_lo, lo_bits, eq_hi, consts->pconst, part_ab, s);
  bit_sums<BITS_COLUMNS>(p, z, 1, 64, 64, xo_live, eq_lo, lo_bits, eq_hi, consts->wconst, part_svc, s);
  *nrows = p.groups * p.splits;
}

// ------------------------------------------------------------------ zerocheck skip fold
// a_mlv[x] = sum_{s in bits(a_x)} w[s] via 8 byte tables of the 64 Lagrange weights;
// word w holds rows 2w (lo) and 2w+1 (hi), which is exactly the first multilinear pair.
// Message: g1 = sum_w eq(w) a1 b1, ginf = sum_w eq(w) (a0 + a1)(b0 + b1). The folded
// vectors are not stored: the next round recomputes them from the bits (below).
__global__ void __launch_bounds__(256)
zc_fold_skip_kernel(const F128d* __restrict__ a, const F128d* __restrict__ b, const F128d* __restrict__ w64,
                    uint64_t n_words, const F128d* __restrict__ eq_lo, uint32_t lo_bits,
                    const F128d* __restrict__ eq_hi, F128d* __restrict__ part, FusedPublish pub) {
  __shared__ F128d T[8][256];
  __shared__ F128d sh[32];
  for (uint32_t e = threadIdx.x; e < 2048; e += blockDim.x) {
    uint32_t c = e >> 8, v = e & 255;
    F128d acc = f128_zero();
    for (int k = 0; k < 8; ++k)
      if ((v >> k) & 1) acc += w64[8 * c + k];
    T[c][v] = acc;
  }
  __syncthreads();
  // a piece of a chunk at a time, one word a thread: the vectors that come here are short
  const uint64_t chunk = 1ull << lo_bits;
  F128d G1 = f128_zero(), GI = f128_zero();
  for (uint64_t w0 = (uint64_t)blockIdx.x * blockDim.x; w0 < n_words; w0 += (uint64_t)gridDim.x * blockDim.x) {
    F128d g1 = f128_zero(), gi = f128_zero();
    const uint64_t wi = w0 + threadIdx.x;
    if (wi < n_words) {
      F128d av = a[wi], bv = b[wi];
      F128d a0 = f128_zero(), a1 = f128_zero(), b0 = f128_zero(), b1 = f128_zero();
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        a0 += T[c][(av.lo >> (8 * c)) & 255];
        a1 += T[c][(av.hi >> (8 * c)) & 255];
        b0 += T[c][(bv.lo >> (8 * c)) & 255];
        b1 += T[c][(bv.hi >> (8 * c)) & 255];
      }
      F128d e = eq_lo[wi & (chunk - 1)];
      g1 = mul_call(e, mul_call(a1, b1));
      gi = mul_call(e, mul_call(a0 + a1, b0 + b1));
    }
    g1 = block_xor(g1, sh);
    gi = block_xor(gi, sh);
    if (threadIdx.x == 0) {
      F128d h = eq_hi ? eq_hi[w0 >> lo_bits] : f128_one();
      G1 += h * g1;
      GI += h * gi;
    }
  }
  if (threadIdx.x == 0) { part[blockIdx.x * 2] = G1; part[blockIdx.x * 2 + 1] = GI; }
  publish_if_last(part, 2, pub, sh);
}
// ---- the weighted form of the zerocheck rounds
// The eq factor of a message over words is eq_lo(low coordinates) * h(chunk), a chunk being
// the 2^LO words that share the high coordinates. a enters every message linearly
// and comes out of tables of the weights, so h is multiplied into a's tables once per chunk:
// the vector kept is a~ = h a, which folds over the low coordinates like a does. eq_lo is left
// to the end: a thread's words (later its pairs) have low indices that do not change from
// chunk to chunk, so it sums a~ b per low index and multiplies each sum by eq_lo once. What is
// left of a message are its two products of variables; the plain form has four (and the
// table form before took two of them from byte tables rebuilt for every 1024 words). When the
// low coordinates are used up, the fold divides by h once (pair_fold's `unweight`), which needs
// every high coordinate to differ from 0 and 1; otherwise the plain form runs.
// All lookups are from window tables (wintable.cuh). Keccak-f 2^18 (87 M live words): skip fold
// 8.05 -> 5.59 ms, folds 12.4 -> 8.4; SHA-256 2^16: 1.25 -> 0.88, 2.25 -> 1.64; BLAKE3 2^12: 83 ->
// 61 us, 0.39 -> 0.37 ms. While a chunk is summed, its threads' next words are on their way and
// the images that the next chunk's table is built from are formed (one barrier and a product's
// latency less a chunk): skip fold 5.55 -> 5.31, folds 8.22 -> 7.88; SHA-256 2^16 0.877 -> 0.841,
// 1.468 -> 1.409.
//
// Skip fold: tables of h w64 (for a) and w64 (for b), six-bit windows, 2 x 82 KB, one block per
// SM; 44 lookups (5.5 cycles of the shared-memory pipe) and two products (13 of the multiply
// pipe) a word.
constexpr uint32_t ZC_W_THREADS = 512;
template <int LO>
__global__ void __launch_bounds__(ZC_W_THREADS, 1)
zc_fold_skip_weighted_kernel(const F128d* __restrict__ a, const F128d* __restrict__ b, const F128d* __restrict__ w64,
                             uint64_t n_chunks, uint64_t n_words, const F128d* __restrict__ eq_lo,
                             const F128d* __restrict__ h, F128d* __restrict__ part, FusedPublish pub) {
  constexpr uint32_t PER = (1u << LO) / ZC_W_THREADS;
  extern __shared__ __align__(16) char wt[];  // a's table, then b's
  __shared__ F128d img[2][64];  // the images of this chunk's table, and the next one's
  __shared__ F128d sh[32];
  const uint32_t lane = win_lane(), team = threadIdx.x >> 3, teams = ZC_W_THREADS / 8;
  char* TB = wt + WinMap<6, 64>::BYTES;
  build_win_map<6, 64>(w64, TB, team, teams);
  F128d S1[PER], SI[PER];
#pragma unroll
  for (uint32_t k = 0; k < PER; ++k) S1[k] = SI[k] = f128_zero();
  auto scale = [&](uint64_t ch, uint32_t buf) {
    if (threadIdx.x < 64 && ch < n_chunks) img[buf][threadIdx.x] = mul_call(h[ch], w64[threadIdx.x]);
  };
  // a thread's words, the next pair of them on its way while this one is summed
  F128d an = f128_zero(), bn = f128_zero();
  auto load = [&](uint64_t wi) {
    if (wi < n_words) { an = a[wi]; bn = b[wi]; }
  };
  scale(blockIdx.x, 0);
  load(((uint64_t)blockIdx.x << LO) + threadIdx.x);
  uint32_t buf = 0;
  for (uint64_t ch = blockIdx.x; ch < n_chunks; ch += gridDim.x, buf ^= 1) {
    __syncthreads();  // the previous chunk's table is no longer read, this one's images are there
    build_win_map<6, 64>(img[buf], wt, team, teams);
    __syncthreads();
    scale(ch + gridDim.x, buf ^ 1);
    const uint64_t w0 = (ch << LO) + threadIdx.x;
#pragma unroll
    for (uint32_t k = 0; k < PER; ++k) {
      const uint64_t wi = w0 + k * ZC_W_THREADS;
      const F128d av = an, bv = bn;
      load(k + 1 < PER ? wi + ZC_W_THREADS : ((ch + gridDim.x) << LO) + threadIdx.x);
      if (wi >= n_words) continue;  // a zero tail
      F128d a0 = f128_zero(), a1 = f128_zero(), b0 = f128_zero(), b1 = f128_zero();
      add_win_map64<6>(a1, av.hi, wt, lane);
      add_win_map64<6>(b1, bv.hi, TB, lane);
      S1[k] += mul_call(a1, b1);
      add_win_map64<6>(a0, av.lo, wt, lane);
      add_win_map64<6>(b0, bv.lo, TB, lane);
      SI[k] += mul_call(a0 + a1, b0 + b1);
    }
  }
  F128d G1 = f128_zero(), GI = f128_zero();
#pragma unroll
  for (uint32_t k = 0; k < PER; ++k) {
    const F128d e = eq_lo[threadIdx.x + k * ZC_W_THREADS];
    G1 += mul_call(e, S1[k]);
    GI += mul_call(e, SI[k]);
  }
  G1 = block_xor(G1, sh);
  GI = block_xor(GI, sh);
  if (threadIdx.x == 0) { part[blockIdx.x * 2] = G1; part[blockIdx.x * 2 + 1] = GI; }
  publish_if_last(part, 2, pub, sh);
}
template <int LO>
static uint32_t fold_skip_weighted(const F128d* a, const F128d* b, const F128d* w64, uint64_t n_words,
                                   const F128d* eq_lo, const F128d* h, F128d* part, cudaStream_t s, FusedPublish pub) {
  const uint64_t n_chunks = (n_words + (1ull << LO) - 1) >> LO;
  const uint32_t blocks = (uint32_t)std::min<uint64_t>(n_chunks, (uint64_t)sm_count());
  const int smem = 2 * WinMap<6, 64>::BYTES;
  set_dynamic_smem((const void*)zc_fold_skip_weighted_kernel<LO>, smem);
  zc_fold_skip_weighted_kernel<LO><<<blocks, ZC_W_THREADS, smem, s>>>(a, b, w64, n_chunks, n_words, eq_lo, h, part, pub);
  LAUNCH_OK();
  return blocks;
}
uint32_t launch_zc_fold_skip_weighted(const F128d* a, const F128d* b, const F128d* w64, uint64_t n_words,
                                      uint32_t lo_bits, const F128d* eq_lo, const F128d* h, F128d* part,
                                      cudaStream_t s, FusedPublish pub) {
  if (lo_bits == 12) return fold_skip_weighted<12>(a, b, w64, n_words, eq_lo, h, part, s, pub);
  if (lo_bits == 11) return fold_skip_weighted<11>(a, b, w64, n_words, eq_lo, h, part, s, pub);
  return fold_skip_weighted<10>(a, b, w64, n_words, eq_lo, h, part, s, pub);
}
uint32_t launch_zc_fold_skip(const F128d* a, const F128d* b, const F128d* w64, uint64_t n_words, const F128d* eq_lo,
                             uint32_t lo_bits, const F128d* eq_hi, F128d* part, cudaStream_t s, FusedPublish pub) {
  const uint32_t blocks = (uint32_t)std::min<uint64_t>((n_words + 255) / 256, (uint64_t)sm_count() * 8);
  zc_fold_skip_kernel<<<blocks, 256, 0, s>>>(a, b, w64, n_words, eq_lo, lo_bits, eq_hi, part, pub);
  LAUNCH_OK();
  return blocks;
}

// The first multilinear fold at rho straight from the bits: the skip-folded pair of word
// w is (sum_s lo_s w_s, sum_s hi_s w_s), so its fold is
//   A'[w] = sum_s lo_s (1 + rho) w_s + sum_s hi_s rho w_s,
// two byte-table sums with the weights pre-scaled by (1 + rho) and rho (no per-word
// multiply). Then the next message over the pairs (A'[2j], A'[2j+1]) with eq(j).
__global__ void zc_scaled_tables_kernel(const F128d* __restrict__ w64, F128d rho, F128d* __restrict__ tabs) {
  __shared__ F128d ws[2][64];
  if (threadIdx.x < 64) {
    F128d v = rho * w64[threadIdx.x];
    ws[1][threadIdx.x] = v;                    // rho * w
    ws[0][threadIdx.x] = v + w64[threadIdx.x];  // (1 + rho) * w
  }
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < 2 * 2048; e += blockDim.x) {
    uint32_t t = e >> 11, c = (e >> 8) & 7, v = e & 255;
    F128d acc = f128_zero();
    for (int k = 0; k < 8; ++k)
      if ((v >> k) & 1) acc += ws[t][8 * c + k];
    tabs[e] = acc;
  }
}
__global__ void __launch_bounds__(256)
zc_fold2_kernel(const F128d* __restrict__ a, const F128d* __restrict__ b, const F128d* __restrict__ tabs,
                uint64_t n_pairs, uint64_t live_pairs, const F128d* __restrict__ eq_lo, uint32_t lo_bits,
                const F128d* __restrict__ eq_hi, F128d* __restrict__ aout, F128d* __restrict__ bout,
                F128d* __restrict__ part, FusedPublish pub) {
  extern __shared__ __align__(16) F128d T[];  // [2][8][256]: (1 + rho) w tables, then rho w tables
  __shared__ F128d sh[32];
  for (uint32_t e = threadIdx.x; e < 4096; e += blockDim.x) T[e] = tabs[e];
  __syncthreads();
  const F128d* T0 = T;
  const F128d* T1 = T + 2048;
  const uint64_t chunk = 1ull << lo_bits;
  const uint64_t n_chunks = (n_pairs + chunk - 1) / chunk;
  F128d G1 = f128_zero(), GI = f128_zero();
  for (uint64_t ch = blockIdx.x; ch < n_chunks; ch += gridDim.x) {
    F128d g1 = f128_zero(), gi = f128_zero();
    uint64_t end = min(n_pairs, (ch + 1) * chunk);
    for (uint64_t j = ch * chunk + threadIdx.x; j < end; j += blockDim.x) {
      if (j >= live_pairs) {  // zero words: zero outputs, nothing added to the message
        aout[2 * j] = aout[2 * j + 1] = bout[2 * j] = bout[2 * j + 1] = f128_zero();
        continue;
      }
      F128d A[2], B[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        F128d av = a[2 * j + h], bv = b[2 * j + h];
        F128d sa = f128_zero(), sb = f128_zero();
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          sa += T0[c * 256 + ((av.lo >> (8 * c)) & 255)] + T1[c * 256 + ((av.hi >> (8 * c)) & 255)];
          sb += T0[c * 256 + ((bv.lo >> (8 * c)) & 255)] + T1[c * 256 + ((bv.hi >> (8 * c)) & 255)];
        }
        A[h] = sa;
        B[h] = sb;
      }
      aout[2 * j] = A[0]; aout[2 * j + 1] = A[1];
      bout[2 * j] = B[0]; bout[2 * j + 1] = B[1];
      F128d e = eq_lo[j & (chunk - 1)];
      g1 += mul_call(e, mul_call(A[1], B[1]));
      gi += mul_call(e, mul_call(A[0] + A[1], B[0] + B[1]));
    }
    g1 = block_xor(g1, sh);
    gi = block_xor(gi, sh);
    if (threadIdx.x == 0) {
      F128d hh = eq_hi ? eq_hi[ch] : f128_one();
      G1 += hh * g1;
      GI += hh * gi;
    }
  }
  if (threadIdx.x == 0) { part[blockIdx.x * 2] = G1; part[blockIdx.x * 2 + 1] = GI; }
  publish_if_last(part, 2, pub, sh);
}
uint32_t launch_zc_fold2(const F128d* a, const F128d* b, const F128d* w64, F128d rho, F128d* tabs, uint64_t n_pairs,
                         uint64_t live_pairs, const F128d* eq_lo, uint32_t lo_bits, const F128d* eq_hi, F128d* aout,
                         F128d* bout, F128d* part, cudaStream_t s, FusedPublish pub) {
  live_pairs = std::min(live_pairs, n_pairs);
  zc_scaled_tables_kernel<<<16, 256, 0, s>>>(w64, rho, tabs);
  LAUNCH_OK();
  set_dynamic_smem((const void*)zc_fold2_kernel, 4096 * 16);
  uint64_t n_chunks = (n_pairs + (1ull << lo_bits) - 1) >> lo_bits;
  uint32_t blocks = (uint32_t)std::min<uint64_t>(n_chunks, (uint64_t)sm_count() * 3);
  zc_fold2_kernel<<<blocks, 256, 4096 * 16, s>>>(a, b, tabs, n_pairs, live_pairs, eq_lo, lo_bits, eq_hi, aout, bout,
                                                  part, pub);
  LAUNCH_OK();
  return blocks;
}

// The weighted form of the first fold (see above): per chunk the tables of h (1 + rho) w and
// h rho w for a, once per block those of (1 + rho) w and rho w for b, five-bit windows, 4 x 50
// KB, one block per SM; 104 lookups (13 cycles) and two products (13) a pair.
template <int LO>
__global__ void __launch_bounds__(ZC_W_THREADS, 1)
zc_fold2_weighted_kernel(const F128d* __restrict__ a, const F128d* __restrict__ b, const F128d* __restrict__ w64,
                         F128d rho, uint64_t n_pairs, uint64_t live_pairs, const F128d* __restrict__ eq_lo,
                         const F128d* __restrict__ h, F128d* __restrict__ aout, F128d* __restrict__ bout,
                         F128d* __restrict__ part, FusedPublish pub) {
  constexpr uint32_t PAIRS = 1u << (LO - 1), PER = PAIRS / ZC_W_THREADS, TAB = WinMap<5, 64>::BYTES;
  extern __shared__ __align__(16) char wt[];  // a's tables for the low and high halves, then b's
  __shared__ F128d wr[2][64], img[2][2][64];  // images of this chunk's tables, and the next one's
  __shared__ F128d sh[32];
  const uint32_t lane = win_lane();
  // two halves of the block build the two tables of a vector
  const uint32_t half = threadIdx.x >= ZC_W_THREADS / 2, team = (threadIdx.x & (ZC_W_THREADS / 2 - 1)) >> 3,
                 teams = ZC_W_THREADS / 16;
  if (threadIdx.x < 64) {
    const F128d v = mul_call(rho, w64[threadIdx.x]);
    wr[1][threadIdx.x] = v;                    // rho w
    wr[0][threadIdx.x] = v + w64[threadIdx.x];  // (1 + rho) w
  }
  __syncthreads();
  build_win_map<5, 64>(wr[half], wt + (2 + half) * TAB, team, teams);
  F128d S1[PER], SI[PER];
#pragma unroll
  for (uint32_t k = 0; k < PER; ++k) S1[k] = SI[k] = f128_zero();
  const uint64_t n_chunks = (n_pairs + PAIRS - 1) / PAIRS;
  auto scale = [&](uint64_t ch, uint32_t buf) {
    if (threadIdx.x < 128 && ch < n_chunks)
      img[buf][threadIdx.x >> 6][threadIdx.x & 63] = mul_call(h[ch], wr[threadIdx.x >> 6][threadIdx.x & 63]);
  };
  // a pair's words, the next pair's on their way while this one is folded
  F128d an[2], bn[2];
  auto load = [&](uint64_t j) {
    if (j >= live_pairs) return;
#pragma unroll
    for (int q = 0; q < 2; ++q) { an[q] = a[2 * j + q]; bn[q] = b[2 * j + q]; }
  };
  an[0] = an[1] = bn[0] = bn[1] = f128_zero();
  scale(blockIdx.x, 0);
  load((uint64_t)blockIdx.x * PAIRS + threadIdx.x);
  uint32_t buf = 0;
  for (uint64_t ch = blockIdx.x; ch < n_chunks; ch += gridDim.x, buf ^= 1) {
    const bool live = ch * PAIRS < live_pairs;  // block-uniform
    if (live) {
      __syncthreads();  // the previous chunk's tables are no longer read, this one's images are there
      build_win_map<5, 64>(img[buf][half], wt + half * TAB, team, teams);
      __syncthreads();
      scale(ch + gridDim.x, buf ^ 1);
    }
#pragma unroll
    for (uint32_t k = 0; k < PER; ++k) {
      const uint64_t j = ch * PAIRS + threadIdx.x + k * ZC_W_THREADS;
      if (j >= n_pairs) continue;
      if (j >= live_pairs) {  // zero words: zero outputs, nothing added to the message
        aout[2 * j] = aout[2 * j + 1] = bout[2 * j] = bout[2 * j + 1] = f128_zero();
        continue;
      }
      F128d A[2] = {an[0], an[1]}, B[2] = {bn[0], bn[1]};
      load(k + 1 < PER ? j + ZC_W_THREADS : (ch + gridDim.x) * PAIRS + threadIdx.x);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const F128d av = A[q], bv = B[q];
        A[q] = B[q] = f128_zero();
        add_win_map64<5>(A[q], av.lo, wt, lane);
        add_win_map64<5>(A[q], av.hi, wt + TAB, lane);
        add_win_map64<5>(B[q], bv.lo, wt + 2 * TAB, lane);
        add_win_map64<5>(B[q], bv.hi, wt + 3 * TAB, lane);
        aout[2 * j + q] = A[q];
        bout[2 * j + q] = B[q];
      }
      S1[k] += mul_call(A[1], B[1]);
      SI[k] += mul_call(A[0] + A[1], B[0] + B[1]);
    }
  }
  F128d G1 = f128_zero(), GI = f128_zero();
#pragma unroll
  for (uint32_t k = 0; k < PER; ++k) {
    const F128d e = eq_lo[threadIdx.x + k * ZC_W_THREADS];
    G1 += mul_call(e, S1[k]);
    GI += mul_call(e, SI[k]);
  }
  G1 = block_xor(G1, sh);
  GI = block_xor(GI, sh);
  if (threadIdx.x == 0) { part[blockIdx.x * 2] = G1; part[blockIdx.x * 2 + 1] = GI; }
  publish_if_last(part, 2, pub, sh);
}
template <int LO>
static uint32_t fold2_weighted(const F128d* a, const F128d* b, const F128d* w64, F128d rho, uint64_t n_pairs,
                               uint64_t live_pairs, const F128d* eq_lo, const F128d* h, F128d* aout, F128d* bout,
                               F128d* part, cudaStream_t s, FusedPublish pub) {
  const int smem = 4 * WinMap<5, 64>::BYTES;
  set_dynamic_smem((const void*)zc_fold2_weighted_kernel<LO>, smem);
  const uint32_t blocks = (uint32_t)std::min<uint64_t>((n_pairs + (1ull << (LO - 1)) - 1) >> (LO - 1), (uint64_t)sm_count());
  zc_fold2_weighted_kernel<LO><<<blocks, ZC_W_THREADS, smem, s>>>(a, b, w64, rho, n_pairs, live_pairs, eq_lo, h, aout,
                                                                  bout, part, pub);
  LAUNCH_OK();
  return blocks;
}
uint32_t launch_zc_fold2_weighted(const F128d* a, const F128d* b, const F128d* w64, F128d rho, uint64_t n_pairs,
                                  uint64_t live_pairs, uint32_t lo_bits, const F128d* eq_lo, const F128d* h,
                                  F128d* aout, F128d* bout, F128d* part, cudaStream_t s, FusedPublish pub) {
  live_pairs = std::min(live_pairs, n_pairs);
  if (lo_bits == 12) return fold2_weighted<12>(a, b, w64, rho, n_pairs, live_pairs, eq_lo, h, aout, bout, part, s, pub);
  if (lo_bits == 11) return fold2_weighted<11>(a, b, w64, rho, n_pairs, live_pairs, eq_lo, h, aout, bout, part, s, pub);
  return fold2_weighted<10>(a, b, w64, rho, n_pairs, live_pairs, eq_lo, h, aout, bout, part, s, pub);
}
// out[c] = prod_j (bit j of c ? f[2j + 1] : f[2j]), j < n: the reciprocals of an eq table from
// those of its factors.
__global__ void factor_table_kernel(const F128d* __restrict__ f, uint32_t n, F128d* __restrict__ out) {
  const uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= (1ull << n)) return;
  F128d v = f128_one();
  for (uint32_t j = 0; j < n; ++j) v = mul_call(v, f[2 * j + ((c >> j) & 1)]);
  out[c] = v;
}
void launch_factor_table(const F128d* f, uint32_t n, F128d* out, cudaStream_t s) {
  factor_table_kernel<<<(unsigned)(((1ull << n) + 255) / 256), 256, 0, s>>>(f, n, out);
  LAUNCH_OK();
}

// ------------------------------------------------------------------ pair fold + message
// Fold the low variable of two vectors at r (out[i] = in[2i] + r (in[2i+1] + in[2i])) and emit
// the pair message over the folded vectors:
//   g1 = sum_j eq(j) A1 B1, ginf = sum_j eq(j) (A0 + A1)(B0 + B1), (A0, A1) = out[2j..2j+2).
// n_pairs = output length / 2 (>= 1); eq by mode (PairEq, plan.h).
// Folds of at least PAIR_FOLD_TABLE_MIN_PAIRS pairs take their products by r from the window table of r (six
// bits, 169 KB, one block per SM): four table products (11 cycles of the shared-memory pipe)
// beside the message's two products of variables (13 of the multiply pipe). The byte tables it
// replaced (three 256-thread blocks per SM) took 4.8 ms for the merged open's rounds of Keccak-f
// 2^18, this form 3.36 (3.53 with a thread on a whole message pair, whose loads 64 bytes apart
// took a quarter of the data pipe, and without the next entries' loads ahead; SHA-256 2^16 0.74 ->
// 0.67). Below the threshold a block would fold less than two rounds of its threads.
template <int EQ>
__global__ void __launch_bounds__(PAIR_FOLD_TABLE_THREADS, 1)
pair_fold_tbl_kernel(const F128d* __restrict__ ain, const F128d* __restrict__ bin, uint64_t n_pairs, uint64_t live_pairs,
                     F128d r, const F128d* __restrict__ eq_lo, uint32_t lo_bits, F128d* __restrict__ aout,
                     F128d* __restrict__ bout, F128d* __restrict__ part, FusedPublish pub) {
  extern __shared__ __align__(16) char wt[];  // WinTable<6>
  __shared__ F128d sh[32];
  build_win_table<6>(r, wt);
  __syncthreads();
  const uint32_t lane = win_lane();
  // A warp takes 32 message pairs, 64 folded entries: lane l folds entries l and 32 + l (two neighbours
  // in memory each), then trades one of them with the lane beside it, so that an even lane has
  // the pair l / 2 and an odd one the pair 16 + l / 2.
  const uint32_t l = threadIdx.x & 31, odd = l & 1;
  const uint64_t w0 = ((uint64_t)blockIdx.x * PAIR_FOLD_TABLE_THREADS + threadIdx.x) >> 5;
  const uint64_t j0 = 32 * w0 + (l >> 1) + 16 * odd, n_warps = (uint64_t)gridDim.x * (PAIR_FOLD_TABLE_THREADS / 32);
  MulAcc m1, mi;
  auto trade = [&](F128d v) {
    return f128(__shfl_xor_sync(0xffffffffu, v.lo, 1), __shfl_xor_sync(0xffffffffu, v.hi, 1));
  };
  F128d xn[4], yn[4];  // the next entries' words
  auto load = [&](uint64_t w) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const uint64_t e = 64 * w + l + 32 * q;
      xn[2 * q] = xn[2 * q + 1] = yn[2 * q] = yn[2 * q + 1] = f128_zero();
      if (e < 2 * live_pairs) {
        xn[2 * q] = ain[2 * e]; xn[2 * q + 1] = ain[2 * e + 1];
        yn[2 * q] = bin[2 * e]; yn[2 * q + 1] = bin[2 * e + 1];
      }
    }
  };
  load(w0);
  for (uint64_t w = w0; 32 * w < n_pairs; w += n_warps) {
    const uint64_t e0 = 64 * w + l;
    F128d A[2], B[2];
    if (32 * w < live_pairs) {  // warp-uniform
      F128d x[4], y[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) { x[q] = xn[q]; y[q] = yn[q]; }
      load(w + n_warps);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        A[q] = x[2 * q] + mul_win<6>(x[2 * q + 1] + x[2 * q], wt, lane);
        B[q] = y[2 * q] + mul_win<6>(y[2 * q + 1] + y[2 * q], wt, lane);
        if (e0 + 32 * q < 2 * n_pairs) {
          aout[e0 + 32 * q] = A[q];
          bout[e0 + 32 * q] = B[q];
        }
      }
      const F128d ta = trade(odd ? A[0] : A[1]), tb = trade(odd ? B[0] : B[1]);
      const F128d A0 = odd ? ta : A[0], A1 = odd ? A[1] : ta, B0 = odd ? tb : B[0], B1 = odd ? B[1] : tb;
      m1.add(A1, B1);
      mi.add(A0 + A1, B0 + B1);
    } else {  // zero inputs: zero outputs, nothing added to the message
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (e0 + 32 * q < 2 * n_pairs) aout[e0 + 32 * q] = bout[e0 + 32 * q] = f128_zero();
    }
  }
  F128d g1 = m1.value(), gi = mi.value();
  if (EQ == EQ_FIXED) {
    const F128d e = eq_lo[j0 & ((1ull << lo_bits) - 1)];
    g1 = mul_call(e, g1);
    gi = mul_call(e, gi);
  }
  g1 = block_xor(g1, sh);
  gi = block_xor(gi, sh);
  if (threadIdx.x == 0) { part[blockIdx.x * 2] = g1; part[blockIdx.x * 2 + 1] = gi; }
  publish_if_last(part, 2, pub, sh);
}
// Small rounds are bound by the latency of a chain of products (a product is about 400
// instructions, and a warp alone on its scheduler issues one every few cycles), so a block takes
// 64 pairs with 256 threads and every thread forms one product at a time: four folds a pair,
// then the two message products beside eq(j) where it is split, then the product by eq. Three
// products deep instead of ten in one thread (14 -> 9 us a round under the profiler; zerocheck folds
// of BLAKE3 2^12 0.35 -> 0.255 ms). Where the two vectors' entries of a pair lie:
// PAIRS (4j .. 4j + 3 in, 2j and 2j + 1 out) or TOP (the top variable bound in place, for the
// lincheck: i, i + h; i + q, i + q + h in, i and i + q out, h = 2q = half the length).
// unweight (or null): factors of the folded a entries. Four blocks a SM: without the bound the walk
// over a grid's pairs takes 70 registers and leaves three.
constexpr uint32_t SMALL_THREADS = 4 * SMALL_PAIRS;
enum PairMap : int { MAP_PAIRS, MAP_TOP };
template <int EQ, int MAP>
__global__ void __launch_bounds__(SMALL_THREADS, 4)
pair_fold_small_kernel(const F128d* ain, const F128d* bin, uint64_t n_pairs, uint64_t live_pairs, F128d r,
                       const F128d* __restrict__ eq_lo, uint32_t lo_bits, const F128d* __restrict__ eq_hi,
                       const F128d* __restrict__ unweight, F128d* aout, F128d* bout, F128d* __restrict__ part,
                       FusedPublish pub) {
  __shared__ F128split rs;  // the fold challenge, split once
  __shared__ F128d v[4][SMALL_PAIRS];  // A0, A1, B0, B1
  __shared__ F128d ev[SMALL_PAIRS];    // eq(j)
  __shared__ F128d sh[SMALL_THREADS / 32];
  if (threadIdx.x == 0) rs = split_factor(r);
  const uint32_t p = threadIdx.x % SMALL_PAIRS, job = threadIdx.x / SMALL_PAIRS;  // whole warps share a job
  F128d acc = f128_zero();
  for (uint64_t base = (uint64_t)blockIdx.x * SMALL_PAIRS; base < n_pairs; base += (uint64_t)gridDim.x * SMALL_PAIRS) {
    {
      // vector a's pairs by the first half of the block, b's by the second; k = 0, 1: out entry
      const uint32_t which = threadIdx.x / (2 * SMALL_PAIRS), i = threadIdx.x % (2 * SMALL_PAIRS);
      const uint32_t q = MAP == MAP_PAIRS ? i >> 1 : i % SMALL_PAIRS, k = MAP == MAP_PAIRS ? i & 1 : i / SMALL_PAIRS;
      const uint64_t j = base + q;
      const F128d* in = which ? bin : ain;
      F128d* out = which ? bout : aout;
      F128d x0 = f128_zero(), d = f128_zero();
      if (j < live_pairs) {
        const uint64_t i0 = MAP == MAP_PAIRS ? 4 * j + 2 * k : j + k * n_pairs;
        x0 = in[i0];
        d = in[MAP == MAP_PAIRS ? i0 + 1 : i0 + 2 * n_pairs] + x0;
      }
      __syncthreads();  // rs is there, the previous pairs' values are no longer read
      F128d f = x0 + mul_split(d, rs);
      const uint64_t o = MAP == MAP_PAIRS ? 2 * j + k : j + k * n_pairs;
      if (unweight && !which && j < live_pairs) f = mul_call(f, unweight[o]);
      if (j < n_pairs) out[o] = f;  // pairs past the live ones have zero inputs
      v[2 * which + k][q] = f;
    }
    __syncthreads();
    F128d t = f128_zero();
    if (job < 2) {
      t = mul_call(job ? v[0][p] + v[1][p] : v[1][p], job ? v[2][p] + v[3][p] : v[3][p]);
    } else if (EQ != EQ_NONE && job == 2) {
      const uint64_t j = min(base + p, n_pairs - 1);
      const F128d lo = eq_lo[j & ((1ull << lo_bits) - 1)];
      ev[p] = EQ == EQ_SPLIT ? mul_call(lo, eq_hi[j >> lo_bits]) : lo;
    }
    if (EQ != EQ_NONE) {
      __syncthreads();
      if (job < 2) t = mul_call(t, ev[p]);
    }
    acc += t;
  }
  acc = warp_xor(acc);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {  // jobs 0 and 1 are two warps each
    part[blockIdx.x * 2] = sh[0] + sh[1];
    part[blockIdx.x * 2 + 1] = sh[2] + sh[3];
  }
  publish_if_last(part, 2, pub, sh);
}
uint32_t launch_pair_fold(const F128d* ain, const F128d* bin, uint64_t n_pairs, uint64_t live_pairs, F128d r,
                          const F128d* eq_lo, uint32_t lo_bits, const F128d* eq_hi, const F128d* unweight, F128d* aout,
                          F128d* bout, F128d* part, cudaStream_t s, FusedPublish pub) {
  live_pairs = std::min(live_pairs, n_pairs);
  const bool fixed = eq_lo && !eq_hi;
  const PairFoldPlan plan =
      pair_fold_plan(n_pairs, eq_hi ? EQ_SPLIT : fixed ? EQ_FIXED : EQ_NONE, lo_bits, unweight != nullptr, (uint64_t)sm_count());
  const uint32_t blocks = plan.blocks;
  if (plan.table) {
    const int smem = WinTable<6>::BYTES;
    if (fixed) {
      set_dynamic_smem((const void*)pair_fold_tbl_kernel<EQ_FIXED>, smem);
      pair_fold_tbl_kernel<EQ_FIXED><<<blocks, PAIR_FOLD_TABLE_THREADS, smem, s>>>(ain, bin, n_pairs, live_pairs, r, eq_lo,
                                                                                   lo_bits, aout, bout, part, pub);
    } else {
      set_dynamic_smem((const void*)pair_fold_tbl_kernel<EQ_NONE>, smem);
      pair_fold_tbl_kernel<EQ_NONE><<<blocks, PAIR_FOLD_TABLE_THREADS, smem, s>>>(ain, bin, n_pairs, live_pairs, r, nullptr,
                                                                                  0, aout, bout, part, pub);
    }
    LAUNCH_OK();
    return blocks;
  }
  auto* kernel = eq_hi ? pair_fold_small_kernel<EQ_SPLIT, MAP_PAIRS>
                       : (fixed ? pair_fold_small_kernel<EQ_FIXED, MAP_PAIRS> : pair_fold_small_kernel<EQ_NONE, MAP_PAIRS>);
  kernel<<<blocks, SMALL_THREADS, 0, s>>>(ain, bin, n_pairs, live_pairs, r, eq_lo, lo_bits, eq_hi, unweight, aout, bout,
                                          part, pub);
  LAUNCH_OK();
  return blocks;
}

// ------------------------------------------------------------------ lincheck
__global__ void lc_eq_inner_kernel(const F128d* __restrict__ w64, const F128d* __restrict__ er, uint32_t K,
                                   F128d* __restrict__ eqi) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < K) eqi[i] = w64[i & 63] * er[i >> 6];
}
void launch_lc_eq_inner(const F128d* w64, const F128d* er, uint32_t K, F128d* eqi, cudaStream_t s) {
  lc_eq_inner_kernel<<<(K + 255) / 256, 256, 0, s>>>(w64, er, K, eqi);
  LAUNCH_OK();
}
// Column folds of A_0 and B_0 (blockIdx.y) in one launch, one warp per column. The matrices are
// dense for sparse ones (BLAKE3 27 M and 17 M entries, SHA-256 29 M and 19 M, columns of up to
// 8943), so a launch is bound by the chain index -> weight of the longest columns and by the
// index traffic: eight loads of each in flight a lane, indices of 16 bits (BLAKE3: two launches of
// 46 us before, one of 74 now).
__global__ void __launch_bounds__(256)
csc_fold_kernel(CscDev A, CscDev B, uint32_t K, const F128d* __restrict__ eqi, F128d* __restrict__ outa,
                F128d* __restrict__ outb) {
  const CscDev& M = blockIdx.y ? B : A;
  F128d* out = blockIdx.y ? outb : outa;
  const uint32_t lane = threadIdx.x & 31, c = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (c >= K) return;
  const uint32_t end = M.col_ptr[c + 1];
  F128d acc = f128_zero();
  uint32_t p = M.col_ptr[c] + lane;
  for (; p + 7 * 32 < end; p += 8 * 32) {
    uint32_t r[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) r[k] = __ldg(M.rows + p + 32 * k);
    F128d v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = eqi[r[k]];
#pragma unroll
    for (int k = 0; k < 8; ++k) acc += v[k];
  }
  for (; p < end; p += 32) acc += eqi[__ldg(M.rows + p)];
  acc = warp_xor(acc);
  if (lane == 0) out[c] = acc;
}
void launch_csc_fold(const CscDev& A, const CscDev& B, uint32_t K, const F128d* eqi, F128d* outa, F128d* outb,
                     cudaStream_t s) {
  csc_fold_kernel<<<dim3((K + 7) / 8, 2), 256, 0, s>>>(A, B, K, eqi, outa, outb);
  LAUNCH_OK();
}

// ---- Keccak-f lincheck columns: ca = eq^T A_0 and cb = eq^T B_0 of the Keccak-f block
// R1CS (the walker of KeccakLincheckCircuit::fold_alpha_batched, crates/flock-prover/src/
// r1cs_hashes/keccak.rs:692-829), as the adjoint of the constraint map. With st_r the
// state before round r and phi = pi o rho o theta, the rows are
//   A[Z] = B[Z] = z_Z;  A[s0] = st_0;  B[s0] = z_Z;  A[s24] = st_24;  B[s24] = z_Z;
//   A[t_r(x,y,z)] = phi(st_r)[x+1,y,z] + z_Z;  B[t_r(x,y,z)] = phi(st_r)[x+2,y,z];
//   st_{r+1} = phi(st_r) + t_r + RC_r z_Z,
// so with lambda_24 = eq[s24] (A) or 0 (B) and, for r = 23..0,
//   column t_r = lambda_{r+1};  lambda_r = phi^T(lambda_{r+1} + eq[t_r] shifted by 1 (A) / 2 (B) in x),
// column s0 = eq[s0] (A only) + lambda_0, and column Z collects eq[Z], the "+ z_Z" rows
// (A: all t rows; B: s0 and s24 rows) and <lambda_{r+1}, RC_r> for every round.
// phi^T = theta^T o (pi o rho)^T:
//   (pi o rho)^T: out[a,b,c] = in[b, 2(a-b) mod 5, c + rho(a,b)]
//   theta^T: out[x,y,z] = in[x,y,z] + sum_y' in[x+1,y',z] + sum_y' in[x-1,y',z+1].
// One block per side, two state words a thread: a thread's lambda stays in its registers, mu goes
// through shared memory (two buffers, so a round has two barriers), every index is formed once and
// the next round's eq weights are on their way while this one is folded. Bound by those 24
// dependent rounds; recomputed indices, four barriers and the loads' latency in each
// made it 131 us a proof.
constexpr uint32_t KW_THREADS = 800, KW_PER = 2;
constexpr uint32_t KW_STATE = KW_THREADS * KW_PER;
constexpr uint32_t KW_S24_WORD = 2048 / 64, KW_T_WORD = 4160 / 64, KW_Z = 4096;
__device__ __forceinline__ uint32_t kw_pos(uint32_t base_word, uint32_t s) { return (base_word + s % 25) * 64 + s / 25; }

__global__ void __launch_bounds__(KW_THREADS)
keccak_lincheck_columns_kernel(const F128d* __restrict__ eqi, F128d* __restrict__ ca, F128d* __restrict__ cb,
                               KeccakColumnConsts kc) {
  extern __shared__ F128d kw_sh[];     // mu of the even, then of the odd rounds
  __shared__ F128d C[320];             // column sums of P = (pi o rho)^T mu: C[x + 5 z]
  __shared__ F128d red[KW_THREADS / 32];
  const bool bside = blockIdx.x == 1;
  F128d* out = bside ? cb : ca;
  const uint32_t shift = bside ? 2 : 1, tid = threadIdx.x;
  F128d zacc = f128_zero();  // this thread's share of column Z beyond eq[Z]
  auto source = [&](uint32_t o) {  // P[o] = mu[source(o)]
    const uint32_t a = o % 5, b = (o / 5) % 5, c = o / 25, y = (2 * (a + 5 - b)) % 5;
    return b + 5 * y + 25 * ((c + kc.rho[a + 5 * b]) & 63);
  };
  F128d lam[KW_PER], e[KW_PER];
  uint32_t own[KW_PER], eqo[KW_PER], src[KW_PER], c1[KW_PER], c2[KW_PER], col[5] = {};
#pragma unroll
  for (uint32_t k = 0; k < KW_PER; ++k) {
    const uint32_t s = tid + k * KW_THREADS, x = s % 5, z = s / 25;
    own[k] = kw_pos(KW_T_WORD, s);                              // columns of t_r: + 1600 r
    eqo[k] = kw_pos(KW_T_WORD, s - x + (x + 5 - shift) % 5);
    src[k] = source(s);
    c1[k] = (x + 1) % 5 + 5 * z;
    c2[k] = (x + 4) % 5 + 5 * ((z + 1) & 63);
    const F128d v = eqi[kw_pos(KW_S24_WORD, s)];
    lam[k] = bside ? f128_zero() : v;
    if (bside) zacc += v;
    e[k] = eqi[eqo[k] + 1600 * 23];
  }
  if (tid < 320)
#pragma unroll
    for (uint32_t y = 0; y < 5; ++y) col[y] = source(tid % 5 + 5 * y + 25 * (tid / 5));
  for (int r = 23; r >= 0; --r) {
    F128d* mu = kw_sh + (r & 1) * KW_STATE;
#pragma unroll
    for (uint32_t k = 0; k < KW_PER; ++k) {
      const uint32_t s = tid + k * KW_THREADS;
      out[own[k] + 1600 * r] = lam[k];
      if (s % 25 == 0 && ((kc.rc[r] >> (s / 25)) & 1)) zacc += lam[k];
      if (!bside) zacc += e[k];
      mu[s] = lam[k] + e[k];
      if (r) e[k] = eqi[eqo[k] + 1600 * (r - 1)];
    }
    __syncthreads();
    if (tid < 320) C[tid] = mu[col[0]] + mu[col[1]] + mu[col[2]] + mu[col[3]] + mu[col[4]];
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < KW_PER; ++k) lam[k] = mu[src[k]] + C[c1[k]] + C[c2[k]];
  }
#pragma unroll
  for (uint32_t k = 0; k < KW_PER; ++k) {
    const uint32_t p = kw_pos(0, tid + k * KW_THREADS);
    const F128d v = eqi[p];
    if (bside) zacc += v;
    out[p] = bside ? lam[k] : lam[k] + v;
  }
  const F128d tot = block_xor(zacc, red);
  if (tid == 0) out[KW_Z] = eqi[KW_Z] + tot;
}
void launch_keccak_lincheck_columns(const F128d* eqi, F128d* ca, F128d* cb, const KeccakColumnConsts& kc,
                                    cudaStream_t s) {
  const int smem = (int)(2 * KW_STATE * sizeof(F128d));
  set_dynamic_smem((const void*)keccak_lincheck_columns_kernel, smem);
  keccak_lincheck_columns_kernel<<<2, KW_THREADS, smem, s>>>(eqi, ca, cb, kc);
  LAUNCH_OK();
}

// The splits' sums of the used columns into zv and its captured copy, zeros in the others.
__global__ void lc_zvec_reduce_kernel(const F128d* __restrict__ part, uint32_t n_split, uint32_t n_out, uint32_t K,
                                      F128d* __restrict__ zv, F128d* __restrict__ captured) {
  uint32_t o = blockIdx.x * blockDim.x + threadIdx.x;  // o = 128 cc + t
  if (o >= K) return;
  F128d acc = f128_zero();
  if (o < n_out) {
    uint32_t cc = o >> 7, t = o & 127;
    for (uint32_t sp = 0; sp < n_split; ++sp) acc += part[((uint64_t)cc * n_split + sp) * 128 + t];
  }
  zv[o] = acc;
  captured[o] = acc;
}
// z_vec[128 cc + t] = sum_row eq(row) * bit_t(z[(cc << nu) + row]).
void launch_lc_zvec(const F128d* z, uint32_t nu, uint32_t used_chunks, const F128d* eq_lo, uint32_t lo_bits,
                    const F128d* eq_hi, F128d* part, uint64_t part_cap, uint32_t K, F128d* zv, F128d* captured,
                    cudaStream_t s) {
  const uint64_t rows = 1ull << nu;
  const BitSumPlan p = bit_sum_plan(used_chunks, rows, part_cap / (used_chunks * 128ull), (uint64_t)sm_count());
  bit_sums<BITS_RAW>(p, z, rows, 1, used_chunks, rows, eq_lo, lo_bits, eq_hi, nullptr, part, s);
  lc_zvec_reduce_kernel<<<(K + 127) / 128, 128, 0, s>>>(part, p.splits, used_chunks * 128, K, zv, captured);
  LAUNCH_OK();
}

// comb = alpha comb_a + comb_b (+ beta at pin); message over the top variable:
//   e1 = sum_i comb[h+i] zv[h+i], einf = sum_i (comb[h+i] + comb[i]) (zv[h+i] + zv[i]).
__global__ void lc_start_kernel(const F128d* __restrict__ ca, const F128d* __restrict__ cb, F128d alpha, F128d beta,
                                uint32_t pin, uint32_t K, F128d* __restrict__ comb, const F128d* __restrict__ zv,
                                F128d* __restrict__ part, FusedPublish pub) {
  __shared__ F128d sh[32];
  uint32_t h = K / 2;
  F128d e1 = f128_zero(), ei = f128_zero();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < h; i += gridDim.x * blockDim.x) {
    F128d c0 = alpha * ca[i] + cb[i], c1 = alpha * ca[i + h] + cb[i + h];
    if (i == pin) c0 += beta;
    if (i + h == pin) c1 += beta;
    comb[i] = c0; comb[i + h] = c1;
    F128d z0 = zv[i], z1 = zv[i + h];
    e1 += c1 * z1;
    ei += (c0 + c1) * (z0 + z1);
  }
  e1 = block_xor(e1, sh);
  ei = block_xor(ei, sh);
  if (threadIdx.x == 0) { part[blockIdx.x * 2] = e1; part[blockIdx.x * 2 + 1] = ei; }
  publish_if_last(part, 2, pub, sh);
}
uint32_t launch_lc_start(const F128d* ca, const F128d* cb, F128d alpha, F128d beta, uint32_t pin, uint32_t K,
                         F128d* comb, const F128d* zv, F128d* part, cudaStream_t s, FusedPublish pub) {
  uint32_t blocks = std::max(1u, std::min((K / 2 + 255) / 256, 256u));
  lc_start_kernel<<<blocks, 256, 0, s>>>(ca, cb, alpha, beta, pin, K, comb, zv, part, pub);
  LAUNCH_OK();
  return blocks;
}
// A union slot's share of the lincheck comb: out[i] = weight (alpha ca[i] + cb[i]), plus
// beta at the slot's const-pin column.
__global__ void lc_slot_comb_kernel(const F128d* __restrict__ ca, const F128d* __restrict__ cb, F128d alpha,
                                    F128d weight, F128d beta, uint32_t pin, uint32_t K, F128d* __restrict__ out) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < K; i += gridDim.x * blockDim.x) {
    F128d c = weight * (alpha * ca[i] + cb[i]);
    if (i == pin) c += beta;
    out[i] = c;
  }
}
void launch_lc_slot_comb(const F128d* ca, const F128d* cb, F128d alpha, F128d weight, F128d beta, uint32_t pin,
                         uint32_t K, F128d* out, cudaStream_t s) {
  lc_slot_comb_kernel<<<std::max(1u, std::min((K + 255) / 256, 1024u)), 256, 0, s>>>(ca, cb, alpha, weight, beta, pin,
                                                                                    K, out);
  LAUNCH_OK();
}
// First top-variable message of a built comb against zv (pairs (i, i + K/2)).
__global__ void lc_top_message_kernel(const F128d* __restrict__ comb, const F128d* __restrict__ zv, uint32_t K,
                                      F128d* __restrict__ part, FusedPublish pub) {
  __shared__ F128d sh[32];
  uint32_t h = K / 2;
  F128d e1 = f128_zero(), ei = f128_zero();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < h; i += gridDim.x * blockDim.x) {
    F128d c0 = comb[i], c1 = comb[i + h], z0 = zv[i], z1 = zv[i + h];
    e1 += c1 * z1;
    ei += (c0 + c1) * (z0 + z1);
  }
  e1 = block_xor(e1, sh);
  ei = block_xor(ei, sh);
  if (threadIdx.x == 0) { part[blockIdx.x * 2] = e1; part[blockIdx.x * 2 + 1] = ei; }
  publish_if_last(part, 2, pub, sh);
}
uint32_t launch_lc_top_message(const F128d* comb, const F128d* zv, uint32_t K, F128d* part, cudaStream_t s, FusedPublish pub) {
  uint32_t blocks = std::max(1u, std::min((K / 2 + 255) / 256, 256u));
  lc_top_message_kernel<<<blocks, 256, 0, s>>>(comb, zv, K, part, pub);
  LAUNCH_OK();
  return blocks;
}

// Bind the top variable of comb and zv (length len -> len/2, in place or not) and emit the next
// top-variable message over the bound vectors (pairs (i, i + len/4)): e1 = sum c1 z1, einf =
// sum (c0 + c1) (z0 + z1).
uint32_t launch_lc_round(const F128d* comb, const F128d* zv, uint32_t len, F128d r, F128d* comb_out, F128d* zv_out,
                         F128d* part, cudaStream_t s, FusedPublish pub) {
  const uint64_t q = len / 4;
  if (q == 0) throw std::runtime_error("lincheck round: fewer than four entries");
  const uint32_t blocks = (uint32_t)((q + SMALL_PAIRS - 1) / SMALL_PAIRS);
  pair_fold_small_kernel<EQ_NONE, MAP_TOP><<<blocks, SMALL_THREADS, 0, s>>>(comb, zv, q, q, r, nullptr, 0, nullptr, nullptr,
                                                                            comb_out, zv_out, part, pub);
  LAUNCH_OK();
  return blocks;
}
// (<w, comb_a>, <w, comb_b>), w[c] = er[c >> 6] * zp[c & 63].
__global__ void lc_matrix_evals_kernel(const F128d* __restrict__ ca, const F128d* __restrict__ cb,
                                       const F128d* __restrict__ er, const F128d* __restrict__ zp, uint32_t K,
                                       F128d* __restrict__ part, FusedPublish pub) {
  __shared__ F128d sh[32];
  F128d ea = f128_zero(), eb = f128_zero();
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < K; c += gridDim.x * blockDim.x) {
    F128d w = er[c >> 6] * zp[c & 63];
    ea += w * ca[c];
    eb += w * cb[c];
  }
  ea = block_xor(ea, sh);
  eb = block_xor(eb, sh);
  if (threadIdx.x == 0) { part[blockIdx.x * 2] = ea; part[blockIdx.x * 2 + 1] = eb; }
  publish_if_last(part, 2, pub, sh);
}
uint32_t launch_lc_matrix_evals(const F128d* ca, const F128d* cb, const F128d* er, const F128d* zp, uint32_t K,
                                F128d* part, cudaStream_t s, FusedPublish pub) {
  uint32_t blocks = std::max(1u, std::min((K + 255) / 256, 256u));
  lc_matrix_evals_kernel<<<blocks, 256, 0, s>>>(ca, cb, er, zp, K, part, pub);
  LAUNCH_OK();
  return blocks;
}
// pub.out[b] = sum_k et[k] * zv[b + 128 k]; one block per b.
__global__ void lc_s_hat_v_kernel(const F128d* __restrict__ zv, const F128d* __restrict__ et, uint32_t n_tail,
                                  FusedPublish pub) {
  __shared__ F128d sh[32];
  uint32_t bb = blockIdx.x;
  F128d acc = f128_zero();
  for (uint32_t k = threadIdx.x; k < n_tail; k += blockDim.x) acc += et[k] * zv[bb + 128 * k];
  acc = block_xor(acc, sh);
  if (threadIdx.x == 0) pub.out[bb] = acc;
  publish_data(pub);
}
void launch_lc_s_hat_v(const F128d* zv, const F128d* et, uint32_t n_tail, cudaStream_t s, FusedPublish pub) {
  lc_s_hat_v_kernel<<<128, 128, 0, s>>>(zv, et, n_tail, pub);
  LAUNCH_OK();
}

// ------------------------------------------------------------------ merged open
// W[d] = sum_c fold_one_slot(er_c[row] * ec_c[col], table_c) for d < area (row = d mod 2^nu,
// col = d >> nu), else 0; round-0 prime over (q, W): u0 = sum q[2i] W[2i],
// u2 = sum (q[2i] + q[2i+1]) (W[2i] + W[2i+1]).
template <bool JAGGED>
__global__ void __launch_bounds__(512, 1)
mo_build_w_kernel(const F128d* __restrict__ q, const F128d* __restrict__ er0, const F128d* __restrict__ ec0,
                  const F128d* __restrict__ er1, const F128d* __restrict__ ec1, const F128d* __restrict__ tables,
                  uint32_t nu, uint64_t area, uint64_t n, F128d* __restrict__ w, F128d* __restrict__ part,
                  JaggedSegs segs, FusedPublish pub) {
  extern __shared__ __align__(16) F128d tab[];  // 2 x 16 x 256
  __shared__ F128d sh[32];
  for (uint32_t i = threadIdx.x; i < 2 * 16 * 256; i += blockDim.x) tab[i] = tables[i];
  __syncthreads();
  const uint64_t rmask = (1ull << nu) - 1;
  F128d u0 = f128_zero(), u2 = f128_zero();
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n / 2; i += (uint64_t)gridDim.x * blockDim.x) {
    if (2 * i >= area) {  // q and W are zero from the area on
      w[2 * i] = w[2 * i + 1] = f128_zero();
      continue;
    }
    F128d W[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      uint64_t d = 2 * i + k;
      F128d acc = f128_zero();
      uint64_t row = d & rmask, col = d >> nu;
      if (d < area && (!JAGGED || jagged_unrank(segs, d, row, col)))
        acc = fold_slot(mul_call(er0[row], ec0[col]), tab) + fold_slot(mul_call(er1[row], ec1[col]), tab + 16 * 256);
      W[k] = acc;
      w[d] = acc;
    }
    F128d q0 = q[2 * i], q1 = q[2 * i + 1];
    u0 += mul_call(q0, W[0]);
    u2 += mul_call(q0 + q1, W[0] + W[1]);
  }
  u0 = block_xor(u0, sh);
  u2 = block_xor(u2, sh);
  if (threadIdx.x == 0) { part[blockIdx.x * 2] = u0; part[blockIdx.x * 2 + 1] = u2; }
  publish_if_last(part, 2, pub, sh);
}
// The same weight under identity compaction with tall columns (col = d >> nu): in column c
// the map x -> fold_slot(x ec_i[c], table_i) is GF(2)-linear, so the block builds its window
// tables (wintable.cuh, five bits, 2 x 101 KB) once per (column, part) work item and W[d] =
// M0_c(er0[row]) + M1_c(er1[row]) is 52 conflict-free lookups and no multiply; only the message's
// products stay integer multiplies. Work item = 2^(nu - part_log) consecutive rows of one column.
// Byte tables (32 lookups, 58 % of their wavefronts conflicts) took 3.60 ms of Keccak-f 2^18, this
// form 3.27; SHA-256 2^16 0.76 -> 0.63.
__global__ void __launch_bounds__(512, 1)
mo_build_w_cols_kernel(const F128d* __restrict__ q, const F128d* __restrict__ er0, const F128d* __restrict__ ec0,
                       const F128d* __restrict__ er1, const F128d* __restrict__ ec1, const F128d* __restrict__ tables,
                       uint32_t nu, uint32_t part_log, uint64_t area, uint64_t n, F128d* __restrict__ w,
                       F128d* __restrict__ part, FusedPublish pub) {
  extern __shared__ __align__(16) char wt[];  // the maps M0, then M1
  __shared__ F128d img[2][128];
  __shared__ F128d sh[32];
  constexpr uint32_t TAB = WinMap<5, 128>::BYTES;
  const uint32_t lane = win_lane(), half = threadIdx.x >> 8;  // two halves of the block build the two tables
  const uint64_t items = (n >> nu) << part_log, rows = 1ull << (nu - part_log);
  MulAcc u0, u2;
  for (uint64_t it = blockIdx.x; it < items; it += gridDim.x) {
    const uint64_t col = it >> part_log, d0 = (col << nu) + ((it & ((1ull << part_log) - 1)) << (nu - part_log));
    const bool used = d0 < area;  // block-uniform
    if (!used) {  // q and W are zero from the area on: zero weights, nothing added to the message
      for (uint64_t j = threadIdx.x; j < rows; j += blockDim.x) w[d0 + j] = f128_zero();
      continue;
    }
    __syncthreads();  // the previous item's tables are no longer read
    if (threadIdx.x < 256) {
      const uint32_t k = threadIdx.x >> 7, t = threadIdx.x & 127;
      img[k][t] = fold_slot(mul_by_power(k ? ec1[col] : ec0[col], t), tables + k * 16 * 256);
    }
    __syncthreads();
    build_win_map<5, 128>(img[half], wt + half * TAB, (threadIdx.x & 255) >> 3, 32);
    __syncthreads();
    for (uint64_t j = threadIdx.x; j < rows / 2; j += blockDim.x) {
      const uint64_t d = d0 + 2 * j, row = d & ((1ull << nu) - 1);
      F128d W0 = f128_zero(), W1 = f128_zero();
      if (d < area) W0 = mul_win<5>(er0[row], wt, lane) + mul_win<5>(er1[row], wt + TAB, lane);
      if (d + 1 < area) W1 = mul_win<5>(er0[row + 1], wt, lane) + mul_win<5>(er1[row + 1], wt + TAB, lane);
      w[d] = W0;
      w[d + 1] = W1;
      const F128d q0 = q[d], q1 = q[d + 1];
      u0.add(q0, W0);
      u2.add(q0 + q1, W0 + W1);
    }
  }
  const F128d r0 = block_xor(u0.value(), sh), r2 = block_xor(u2.value(), sh);
  if (threadIdx.x == 0) { part[blockIdx.x * 2] = r0; part[blockIdx.x * 2 + 1] = r2; }
  publish_if_last(part, 2, pub, sh);
}
// Columns of at least 2^MO_COLS_MIN_NU rows take the column-table form (stage times with and
// without it, BLAKE3 2^11: 65 and 74 us, SHA-256 2^11: 83 and 85, 2^13: 141 and 183).
constexpr uint32_t MO_COLS_MIN_NU = 11;
// A work item's tables cost about as much as 2^10 rows: the split of the columns into 2^part_log
// items each that gives the last block to finish the least to do (SHA-256 2^14 in items of 2^14,
// 2^13 and 2^12 rows: 236, 209 and 230 us).
static uint32_t mo_part_log(uint32_t nu, uint64_t area) {
  uint32_t best = 0;
  uint64_t least = ~0ull;
  for (uint32_t p = 0; nu - p >= 11; ++p) {
    const uint64_t rows = 1ull << (nu - p), items = (area + rows - 1) / rows, sms = (uint64_t)sm_count();
    const uint64_t cost = (items + sms - 1) / sms * (rows + 1024);
    if (cost < least) { least = cost; best = p; }
  }
  return best;
}
uint32_t launch_mo_build_w(const F128d* q, const F128d* er0, const F128d* ec0, const F128d* er1, const F128d* ec1,
                           const F128d* tables, uint32_t nu, uint64_t area, uint64_t n, F128d* w, F128d* part,
                           cudaStream_t s, FusedPublish pub, const JaggedSegs* segs) {
  if (!segs && nu >= MO_COLS_MIN_NU && (n >> nu) >= 1 && (n & ((1ull << nu) - 1)) == 0) {
    const uint32_t part_log = mo_part_log(nu, area);
    const uint64_t items = (n >> nu) << part_log;
    const uint32_t blocks = (uint32_t)std::min<uint64_t>(items, (uint64_t)sm_count());
    const int smem = 2 * WinMap<5, 128>::BYTES;
    set_dynamic_smem((const void*)mo_build_w_cols_kernel, smem);
    mo_build_w_cols_kernel<<<blocks, 512, smem, s>>>(q, er0, ec0, er1, ec1, tables, nu, part_log, area, n, w, part, pub);
    LAUNCH_OK();
    return blocks;
  }
  size_t smem = 2 * 16 * 256 * sizeof(F128d);
  uint32_t blocks = (uint32_t)std::min<uint64_t>((n / 2 + 511) / 512, (uint64_t)sm_count());
  if (segs) {
    set_dynamic_smem((const void*)mo_build_w_kernel<true>, (int)smem);
    mo_build_w_kernel<true><<<blocks, 512, smem, s>>>(q, er0, ec0, er1, ec1, tables, nu, area, n, w, part, *segs, pub);
  } else {
    set_dynamic_smem((const void*)mo_build_w_kernel<false>, (int)smem);
    mo_build_w_kernel<false><<<blocks, 512, smem, s>>>(q, er0, ec0, er1, ec1, tables, nu, area, n, w, part,
                                                       JaggedSegs(), pub);
  }
  LAUNCH_OK();
  return blocks;
}

// ------------------------------------------------------------------ Ligerito
// ---- the lane stage: the first initial_k folds, over the lanes of the committed stack
// q[l * D + p] (lane l, row p < D). The basis there is a sum of terms c_t eq(x_t) over all
// variables, so it is never formed: with the lane dots
//   h_t[l] = sum_p q[l D + p] eq_t(p)
// every message of these folds is a sum over lane pairs (on the host, at most 64 lanes), and
// once all the challenges are known f is folded by all of them in one pass,
//   f[p] = sum_l lambda_l q[l D + p],  lambda = eq(challenges) in F256,
// and the basis is sum_t e_t eq_t(p). This reads q once for the dots and once for the fold.
// Forming the basis and folding both vectors challenge by challenge read and wrote them six
// times: the whole Ligerito stage took 26.4 ms of a Keccak-f 2^18 proof (9.3 with this stage, 8.0 with
// the later changes to the levels), 4.8 ms of SHA-256 2^16 (2.6, 2.0), 0.94 ms of BLAKE3 2^12 (0.69,
// 0.57; six kernels and round trips fewer).

// Lane dots h[l] = sum_p q[l D + p] eq(p), as rows of `lanes` partials.
uint32_t launch_lg_lane_dots(const F128d* q, uint32_t lanes, uint32_t log_d, const F128d* eq_lo, uint32_t lo_bits,
                             const F128d* eq_hi, F128d* part, uint64_t part_room, cudaStream_t s) {
  const uint64_t rows = 1ull << log_d;
  const BitSumPlan p = bit_sum_plan(lanes, rows, BITS_MAX_SPLITS, (uint64_t)sm_count());
  if (uint64_t(p.splits) * lanes > part_room) throw std::runtime_error("lane dots exceed the partials buffer");
  bit_sums<BITS_DOT>(p, q, rows, 1, lanes, rows, eq_lo, lo_bits, eq_hi, nullptr, part, s);
  return p.splits;
}
// The fold of all lanes: part[g D + p] = sum over the lanes of group g of lambda_l q[l D + p].
// A block holds LANE_FOLD_ROWS rows' F256 sums in registers and walks its lanes: per lane the
// window tables of lambda's two halves (W = 5, 202 KB, one block per SM), the next lane's words
// loaded before the tables are built; two products a word, one in four split. Groups split the
// lanes where the rows alone do not fill the SMs; lg_lane_switch sums them.
constexpr uint32_t LANE_FOLD_THREADS = 512, LANE_FOLD_PER = 6;
constexpr uint32_t LANE_FOLD_ROWS = LANE_FOLD_THREADS * LANE_FOLD_PER;
__global__ void __launch_bounds__(LANE_FOLD_THREADS, 1)
lg_lane_fold_kernel(const F128d* __restrict__ q, const F256d* __restrict__ lambda, uint32_t lanes, uint64_t D,
                    F256d* __restrict__ part) {
  extern __shared__ __align__(16) char wt[];  // the WinTable<5> of lambda.c0, then lambda.c1's
  __shared__ F128split s1;
  const uint32_t l0 = lanes * blockIdx.y / gridDim.y, l1 = lanes * (blockIdx.y + 1) / gridDim.y, lane16 = win_lane();
  const uint64_t p0 = (uint64_t)blockIdx.x * LANE_FOLD_ROWS + threadIdx.x;
  F128d c0[LANE_FOLD_PER], c1[LANE_FOLD_PER], x[LANE_FOLD_PER];
#pragma unroll
  for (uint32_t k = 0; k < LANE_FOLD_PER; ++k) {
    const uint64_t p = p0 + k * LANE_FOLD_THREADS;
    c0[k] = c1[k] = f128_zero();
    x[k] = p < D ? q[l0 * D + p] : f128_zero();
  }
  for (uint32_t l = l0; l < l1; ++l) {
    __syncthreads();  // the previous lane's tables are no longer read
    const F256d lam = lambda[l];
    if (threadIdx.x == 0) s1 = split_factor(lam.c1);
    build_win_table<5>(lam.c0, wt);
    build_win_table<5>(lam.c1, wt + WinTable<5>::BYTES);
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < LANE_FOLD_PER; ++k) {
      c0[k] += mul_win<5>(x[k], wt, lane16);
      c1[k] += (k & 1) ? mul_split(x[k], s1) : mul_win<5>(x[k], wt + WinTable<5>::BYTES, lane16);
    }
    if (l + 1 < l1) {
#pragma unroll
      for (uint32_t k = 0; k < LANE_FOLD_PER; ++k) {
        const uint64_t p = p0 + k * LANE_FOLD_THREADS;
        if (p < D) x[k] = q[(l + 1) * D + p];
      }
    }
  }
#pragma unroll
  for (uint32_t k = 0; k < LANE_FOLD_PER; ++k) {
    const uint64_t p = p0 + k * LANE_FOLD_THREADS;
    if (p < D) part[blockIdx.y * D + p] = f256(c0[k], c1[k]);
  }
}
// Lane groups: enough that the grid holds about eight blocks per SM (or a lane a group).
uint32_t lane_fold_groups(uint32_t lanes, uint64_t D, uint64_t sms) {
  const uint64_t rows = (D + LANE_FOLD_ROWS - 1) / LANE_FOLD_ROWS, want = sms * 8;
  return (uint32_t)std::min<uint64_t>(lanes, (want + rows - 1) / rows);
}
void launch_lg_lane_fold(const F128d* q, const F256d* lambda, uint32_t lanes, uint64_t D, F256d* part, cudaStream_t s) {
  const int smem = 2 * WinTable<5>::BYTES;
  set_dynamic_smem((const void*)lg_lane_fold_kernel, smem);
  const dim3 grid((unsigned)((D + LANE_FOLD_ROWS - 1) / LANE_FOLD_ROWS), lane_fold_groups(lanes, D, (uint64_t)sm_count()));
  lg_lane_fold_kernel<<<grid, LANE_FOLD_THREADS, smem, s>>>(q, lambda, lanes, D, part);
  LAUNCH_OK();
}
// Round message with block pairing d: pairs (lo, lo + d), lo = 2 d blk + k.
//   u0 = sum f[lo] b[lo], u2 = sum (f[lo] + f[hi]) (b[lo] + b[hi]),
// four words per block (u0.c0, u0.c1, u2.c0, u2.c1).
// The pairing distances are powers of two (the kernels take log2 d).
static uint32_t log2_distance(uint64_t d) {
  if (d == 0 || (d & (d - 1))) throw std::runtime_error("Ligerito pair distance must be a power of two");
  uint32_t l = 0;
  while ((uint64_t(1) << l) < d) ++l;
  return l;
}
__device__ __forceinline__ uint64_t pair_lo(uint64_t i, uint32_t d_log) {
  return ((i >> d_log) << (d_log + 1)) | (i & ((1ull << d_log) - 1));
}
__global__ void lg_message256_kernel(const F256d* __restrict__ f, const F256d* __restrict__ b, uint64_t n,
                                     uint32_t d_log, F128d* __restrict__ part, FusedPublish pub) {
  __shared__ F128d sh[32];
  F256d u0 = f256(f128_zero(), f128_zero()), u2 = u0;
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n / 2; p += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t lo = pair_lo(p, d_log), hi = lo + (1ull << d_log);
    F256d f0 = f[lo], f1 = f[hi], b0 = b[lo], b1 = b[hi];
    u0 += f256_mul_call(f0, b0);
    u2 += f256_mul_call(f0 + f1, b0 + b1);
  }
  F128d r0 = block_xor(u0.c0, sh), r1 = block_xor(u0.c1, sh), r2 = block_xor(u2.c0, sh), r3 = block_xor(u2.c1, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x * 4] = r0; part[blockIdx.x * 4 + 1] = r1;
    part[blockIdx.x * 4 + 2] = r2; part[blockIdx.x * 4 + 3] = r3;
  }
  if (pub.out) publish_if_last(part, 4, pub, sh);
}
uint32_t launch_lg_message256(const F256d* f, const F256d* b, uint64_t n, uint64_t d, F128d* part,
                              cudaStream_t s, FusedPublish pub) {
  uint32_t blocks = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((n / 2 + 255) / 256, (uint64_t)sm_count() * 8));
  lg_message256_kernel<<<blocks, 256, 0, s>>>(f, b, n, log2_distance(d), part, pub);
  LAUNCH_OK();
  return blocks;
}
__global__ void lg_fold256_kernel(const F256d* __restrict__ f, const F256d* __restrict__ b, uint64_t n_out, F256d r,
                                  uint32_t d_log, F256d* __restrict__ fo, F256d* __restrict__ bo) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_out) return;
  const uint64_t lo = pair_lo(i, d_log), hi = lo + (1ull << d_log);
  F256d f0 = f[lo], b0 = b[lo];
  fo[i] = f0 + f256_mul_call(r, f[hi] + f0);
  bo[i] = b0 + f256_mul_call(r, b[hi] + b0);
}
void launch_lg_fold256(const F256d* f, const F256d* b, uint64_t n_out, F256d r, uint64_t d,
                       F256d* fo, F256d* bo, cudaStream_t s) {
  lg_fold256_kernel<<<(unsigned)((n_out + 255) / 256), 256, 0, s>>>(f, b, n_out, r, log2_distance(d), fo, bo);
  LAUNCH_OK();
}
// One round's fold (at r, pairs d_fold apart) fused with the next round's message over the
// folded vectors (pairs d_msg apart): u0 = sum f0 b0, u2 = sum (f0 + f1)(b0 + b1), same index
// maps as lg_fold256_kernel and lg_message256_kernel.
// Large rounds: the products by r come from byte tables of r.c0 and r.c1 plus the split form of
// r.c0 + r.c1 (the Karatsuba terms of F256 product, see operator* in field.cuh): per pair
// 8 table products on the load/store pipe beside 4 + 6 integer-multiply products. One
// 512-thread block per SM holds the two tables (141 KB).
__global__ void __launch_bounds__(512, 1)
lg_fold_msg256_tbl_kernel(const F256d* __restrict__ f, const F256d* __restrict__ b, uint64_t n_out, F256d r,
                          uint32_t dlog_fold, uint32_t dlog_msg, F256d* __restrict__ fo, F256d* __restrict__ bo,
                          F128d* __restrict__ part, FusedPublish pub) {
  extern __shared__ __align__(16) F128d rtab[];  // tables of r.c0 and r.c1
  __shared__ F128d sh[32];
  __shared__ F128split rsum;
  if (threadIdx.x == 0) rsum = split_factor(r.c0 + r.c1);
  build_byte_table(r.c0, rtab);
  build_byte_table(r.c1, rtab + BYTE_TABLE_ENTRIES);  // its scratch follows the second table
  auto fold = [&](F256d v0, F256d d) {
    const F128d p0 = mul_table(d.c0, rtab), p1 = mul_table(d.c1, rtab + BYTE_TABLE_ENTRIES),
                p2 = mul_split_call(d.c0 + d.c1, &rsum);
    return v0 + f256(p0 + mul_by_x_inv(p1), p2 + p0);
  };
  auto fold_at = [&](uint64_t i, F256d& fi, F256d& bi) {
    const uint64_t lo = pair_lo(i, dlog_fold), hi = lo + (1ull << dlog_fold);
    const F256d f0 = f[lo], b0 = b[lo];
    fi = fold(f0, f[hi] + f0);
    bi = fold(b0, b[hi] + b0);
  };
  F256d u0 = f256(f128_zero(), f128_zero()), u2 = u0;
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n_out / 2; p += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t olo = pair_lo(p, dlog_msg), ohi = olo + (1ull << dlog_msg);
    F256d fl, bl, fh, bh;
    fold_at(olo, fl, bl);
    fo[olo] = fl;
    bo[olo] = bl;
    u0 += f256_mul_call(fl, bl);
    fold_at(ohi, fh, bh);
    fo[ohi] = fh;
    bo[ohi] = bh;
    u2 += f256_mul_call(fl + fh, bl + bh);
  }
  F128d r0 = block_xor(u0.c0, sh), r1 = block_xor(u0.c1, sh), r2 = block_xor(u2.c0, sh), r3 = block_xor(u2.c1, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x * 4] = r0; part[blockIdx.x * 4 + 1] = r1;
    part[blockIdx.x * 4 + 2] = r2; part[blockIdx.x * 4 + 3] = r3;
  }
  publish_if_last(part, 4, pub, sh);
}
// Small rounds (see pair_fold_small_kernel): a block takes 32 message pairs with 384 threads. A
// warp forms one of the 12 products of the four folds (f and b, both entries, the three Karatsuba
// products) for its 32 pairs, then one of the message's six; two products deep instead of
// eighteen in one thread (28 us a round at any size before, 11 now, under the profiler).
constexpr uint32_t LG_SMALL_THREADS = 12 * 32;
__global__ void __launch_bounds__(LG_SMALL_THREADS)
lg_fold_msg256_small_kernel(const F256d* __restrict__ f, const F256d* __restrict__ b, uint64_t n_out, F256d r,
                            uint32_t dlog_fold, uint32_t dlog_msg, F256d* __restrict__ fo, F256d* __restrict__ bo,
                            F128d* __restrict__ part, FusedPublish pub) {
  __shared__ F128split rs[3];     // r.c0, r.c1, r.c0 + r.c1
  __shared__ F128d prod[12][32];
  __shared__ F256d out[4][32];    // f low, b low, f high, b high entry of the pair
  __shared__ F128d sh[32];
  const uint32_t w = threadIdx.x >> 5, t = threadIdx.x & 31, vec = w / 3, comp = w % 3;
  if (threadIdx.x < 3) rs[threadIdx.x] = split_factor(threadIdx.x == 0 ? r.c0 : threadIdx.x == 1 ? r.c1 : r.c0 + r.c1);
  const uint64_t p = (uint64_t)blockIdx.x * 32 + t;
  const bool have = p < n_out / 2;
  auto part_of = [](F256d x, uint32_t c) { return c == 0 ? x.c0 : c == 1 ? x.c1 : x.c0 + x.c1; };
  F256d v0 = f256(f128_zero(), f128_zero()), d = v0;
  uint64_t o = 0;
  if (have) {
    const F256d* in = (vec & 1) ? b : f;
    o = pair_lo(p, dlog_msg) + ((vec >> 1) ? 1ull << dlog_msg : 0);
    const uint64_t lo = pair_lo(o, dlog_fold);
    v0 = in[lo];
    d = in[lo + (1ull << dlog_fold)] + v0;
  }
  __syncthreads();
  const F128d mine = mul_split(part_of(d, comp), rs[comp]);
  prod[w][t] = mine;
  __syncthreads();
  if (comp == 0) {
    const F128d p1 = prod[w + 1][t], p2 = prod[w + 2][t];
    const F256d v = v0 + f256(mine + mul_by_x_inv(p1), p2 + mine);
    if (have) ((vec & 1) ? bo : fo)[o] = v;
    out[vec][t] = v;
  }
  __syncthreads();
  if (w < 6) {
    const uint32_t sum = w / 3;  // u0, then u2
    F256d x = out[0][t], y = out[1][t];
    if (sum) {
      x += out[2][t];
      y += out[3][t];
    }
    const F128d q = warp_xor(mul(part_of(x, comp), part_of(y, comp)));
    if (t == 0) prod[w][0] = q;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t k = 0; k < 2; ++k) {
      const F128d q0 = prod[3 * k][0], q1 = prod[3 * k + 1][0], q2 = prod[3 * k + 2][0];
      part[blockIdx.x * 4 + 2 * k] = q0 + mul_by_x_inv(q1);
      part[blockIdx.x * 4 + 2 * k + 1] = q2 + q0;
    }
  }
  publish_if_last(part, 4, pub, sh);
}
// Folds of at least this many output entries use the table form, with at least
// LG_FOLD_TABLE_MIN_BLOCK_PAIRS message pairs per block for its two table builds.
constexpr uint64_t LG_FOLD_TABLE_MIN_OUT = uint64_t(1) << 17;
constexpr uint64_t LG_FOLD_TABLE_MIN_BLOCK_PAIRS = 512;
uint32_t launch_lg_fold_msg256(const F256d* f, const F256d* b, uint64_t n_out, F256d r, uint64_t d_fold,
                               uint64_t d_msg, F256d* fo, F256d* bo, F128d* part, cudaStream_t s, FusedPublish pub) {
  if (n_out >= LG_FOLD_TABLE_MIN_OUT) {
    const int smem = (int)((BYTE_TABLE_ENTRIES + BYTE_TABLE_SMEM_ENTRIES) * sizeof(F128d));
    set_dynamic_smem((const void*)lg_fold_msg256_tbl_kernel, smem);
    const uint32_t blocks = (uint32_t)std::max<uint64_t>(
        1, std::min<uint64_t>((uint64_t)sm_count(), n_out / 2 / LG_FOLD_TABLE_MIN_BLOCK_PAIRS));
    lg_fold_msg256_tbl_kernel<<<blocks, 512, smem, s>>>(f, b, n_out, r, log2_distance(d_fold), log2_distance(d_msg), fo,
                                                        bo, part, pub);
    LAUNCH_OK();
    return blocks;
  }
  const uint32_t blocks = (uint32_t)std::max<uint64_t>(1, (n_out / 2 + 31) / 32);
  lg_fold_msg256_small_kernel<<<blocks, LG_SMALL_THREADS, 0, s>>>(f, b, n_out, r, log2_distance(d_fold),
                                                                  log2_distance(d_msg), fo, bo, part, pub);
  LAUNCH_OK();
  return blocks;
}
// f' = (f.c0, f.c1) interleaved as base values; b' = (b, u b).
__global__ void lg_code_switch_kernel(const F256d* __restrict__ f, const F256d* __restrict__ b, uint64_t n,
                                      F256d* __restrict__ fo, F256d* __restrict__ bo) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  F256d fv = f[i], bv = b[i];
  fo[2 * i] = f256_base(fv.c0);
  fo[2 * i + 1] = f256_base(fv.c1);
  bo[2 * i] = bv;
  bo[2 * i + 1] = f256(mul_by_x_inv(bv.c1), bv.c0 + bv.c1);
}
void launch_lg_code_switch(const F256d* f, const F256d* b, uint64_t n, F256d* fo, F256d* bo, cudaStream_t s) {
  lg_code_switch_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(f, b, n, fo, bo);
  LAUNCH_OK();
}
// The code switch fused with the next message (pairs (2i, 2i + 1) of the switched vectors).
// The switched f entries are base-field, so both products of pair i are base x F256, two
// F128 products each instead of three:
//   u0 += f.c0 b = (f.c0 b.c0, f.c0 b.c1),
//   u2 += (f.c0 + f.c1)(b + u b) = s (b.c0 + x^-1 b.c1, b.c0),  s = f.c0 + f.c1,
// with u b = (x^-1 b.c1, b.c0 + b.c1) as the switch writes it.
__device__ __forceinline__ void switch_pair(F256d fv, F256d bv, uint64_t i, F256d* __restrict__ fo,
                                            F256d* __restrict__ bo, F128d& u00, F128d& u01, F128d& u20, F128d& u21) {
  const F128d ub0 = mul_by_x_inv(bv.c1);
  fo[2 * i] = f256_base(fv.c0);
  fo[2 * i + 1] = f256_base(fv.c1);
  bo[2 * i] = bv;
  bo[2 * i + 1] = f256(ub0, bv.c0 + bv.c1);
  const F128d sv = fv.c0 + fv.c1;
  u00 += mul_call(fv.c0, bv.c0);
  u01 += mul_call(fv.c0, bv.c1);
  u20 += mul_call(sv, bv.c0 + ub0);
  u21 += mul_call(sv, bv.c0);
}
__device__ __forceinline__ void switch_publish(F128d u00, F128d u01, F128d u20, F128d u21, F128d* __restrict__ part,
                                               const FusedPublish& pub, F128d* sh) {
  const F128d r0 = block_xor(u00, sh), r1 = block_xor(u01, sh), r2 = block_xor(u20, sh), r3 = block_xor(u21, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x * 4] = r0; part[blockIdx.x * 4 + 1] = r1;
    part[blockIdx.x * 4 + 2] = r2; part[blockIdx.x * 4 + 3] = r3;
  }
  if (pub.out) publish_if_last(part, 4, pub, sh);
}
__global__ void lg_switch_msg_kernel(const F256d* __restrict__ f, const F256d* __restrict__ b, uint64_t n,
                                     F256d* __restrict__ fo, F256d* __restrict__ bo, F128d* __restrict__ part,
                                     FusedPublish pub) {
  __shared__ F128d sh[32];
  F128d u00 = f128_zero(), u01 = f128_zero(), u20 = f128_zero(), u21 = f128_zero();
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
    switch_pair(f[i], b[i], i, fo, bo, u00, u01, u20, u21);
  switch_publish(u00, u01, u20, u21, part, pub, sh);
}
uint32_t launch_lg_switch_msg(const F256d* f, const F256d* b, uint64_t n, F256d* fo, F256d* bo, F128d* part,
                              cudaStream_t s, FusedPublish pub) {
  uint32_t blocks = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, (uint64_t)sm_count() * 8));
  lg_switch_msg_kernel<<<blocks, 256, 0, s>>>(f, b, n, fo, bo, part, pub);
  LAUNCH_OK();
  return blocks;
}
// The end of the lane stage: f[p] summed over the fold's lane groups, b[p] = sum_t e_t eq_t(p),
// then the code switch and its message as lg_switch_msg. The live entries are the rows.
__global__ void lg_lane_switch_kernel(const F256d* __restrict__ fpart, uint32_t groups, LaneTerms terms, uint64_t D,
                                      F256d* __restrict__ fo, F256d* __restrict__ bo, F128d* __restrict__ part,
                                      FusedPublish pub) {
  __shared__ F128d sh[32];
  __shared__ F128d scale[2 * LaneTerms::MAX];  // coef_t hi_t of these 256 rows (one entry of hi covers them)
  F128d u00 = f128_zero(), u01 = f128_zero(), u20 = f128_zero(), u21 = f128_zero();
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x; i0 < D; i0 += step) {
    __syncthreads();  // the previous rows' factors are no longer read
    if (threadIdx.x < 2 * terms.n) {
      const uint32_t t = threadIdx.x >> 1;
      scale[threadIdx.x] = mul_call(threadIdx.x & 1 ? terms.coef[t].c1 : terms.coef[t].c0, terms.hi[t][i0 >> terms.lo_bits]);
    }
    __syncthreads();
    const uint64_t i = i0 + threadIdx.x;
    if (i >= D) continue;
    F256d fv = fpart[i], bv = f256(f128_zero(), f128_zero());
#pragma unroll 8
    for (uint32_t g = 1; g < groups; ++g) fv += fpart[g * D + i];
    for (uint32_t t = 0; t < terms.n; ++t) {
      const F128d e = terms.lo[t][i & ((1ull << terms.lo_bits) - 1)];
      bv += f256(mul_call(scale[2 * t], e), mul_call(scale[2 * t + 1], e));
    }
    switch_pair(fv, bv, i, fo, bo, u00, u01, u20, u21);
  }
  switch_publish(u00, u01, u20, u21, part, pub, sh);
}
uint32_t launch_lg_lane_switch(const F256d* fpart, uint32_t groups, const LaneTerms& terms, uint64_t D, F256d* fo,
                               F256d* bo, F128d* part, cudaStream_t s, FusedPublish pub) {
  const uint32_t blocks = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((D + 255) / 256, (uint64_t)sm_count() * 8));
  lg_lane_switch_kernel<<<blocks, 256, 0, s>>>(fpart, groups, terms, D, fo, bo, part, pub);
  LAUNCH_OK();
  return blocks;
}
// mat[i] = f[i mod msg].c0
__global__ void lg_replicate_kernel(const F256d* __restrict__ f, uint64_t msg, uint64_t total, F128d* __restrict__ mat) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < total) mat[i] = f[i & (msg - 1)].c0;
}
void launch_lg_replicate(const F256d* f, uint64_t msg, uint64_t total, F128d* mat, cudaStream_t s) {
  lg_replicate_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(f, msg, total, mat);
  LAUNCH_OK();
}
// Pending eq basis e = eq(z) over the (base-valued) f of length 2 pairs: with t(j) the eq over
// z[1 ..], e[2j] = (1 + z_0) t(j) and e[2j + 1] = z_0 t(j), so the basis is stored as t and the
// message comes from S0 = sum f[2j] t(j), S1 = sum f[2j + 1] t(j), published: three products a
// pair (five with e itself). Up to a size (below) the block forms t's two factors itself, lo of
// eight coordinates an entry a thread, hi for its 256 pairs, and no table launch precedes it.
template <bool TABLES>
__global__ void __launch_bounds__(EQ_THREADS)
lg_intro_eq_kernel(const F256d* __restrict__ f, const F128d* __restrict__ point, uint32_t n_vars,
                   const F128d* __restrict__ eq_lo, uint32_t lo_bits, const F128d* __restrict__ eq_hi, uint64_t pairs,
                   F128d* __restrict__ pend, F128d* __restrict__ part, FusedPublish pub) {
  __shared__ F128d sh[32];
  __shared__ F128d sub[TABLES ? 1 : 2][EQ_MAX_GROUPS][16];
  F128d s0 = f128_zero(), s1 = f128_zero(), lo = f128_one();
  const uint32_t lo_n = min(n_vars, 8u), hi_n = n_vars - lo_n;
  if (!TABLES) {
    eq_sub_tables(point, lo_n, sub[0]);
    eq_sub_tables(point + lo_n, hi_n, sub[TABLES ? 0 : 1]);
    __syncthreads();
    lo = eq_from_sub(sub[0], lo_n, threadIdx.x & ((1u << lo_n) - 1));
  }
  for (uint64_t j = (uint64_t)blockIdx.x * EQ_THREADS + threadIdx.x; j < pairs; j += (uint64_t)gridDim.x * EQ_THREADS) {
    F128d t;
    if (TABLES) t = eq_at(eq_lo, lo_bits, eq_hi, j);
    else t = hi_n ? mul_call(lo, eq_from_sub(sub[TABLES ? 0 : 1], hi_n, j >> 8)) : lo;
    pend[j] = t;
    s0 += mul_call(f[2 * j].c0, t);
    s1 += mul_call(f[2 * j + 1].c0, t);
  }
  s0 = block_xor(s0, sh);
  s1 = block_xor(s1, sh);
  if (threadIdx.x == 0) { part[blockIdx.x * 2] = s0; part[blockIdx.x * 2 + 1] = s1; }
  publish_if_last(part, 2, pub, sh);
}
// One pair a thread of at most four blocks of 256 on each SM.
bool lg_intro_eq_direct(uint64_t pairs) { return pairs <= (uint64_t)sm_count() * 4 * EQ_THREADS; }
void launch_lg_intro_eq(const F256d* f, const F128d* point, uint32_t n_vars, uint64_t pairs, F128d* pend, F128d* part,
                        cudaStream_t s, FusedPublish pub) {
  const uint32_t blocks = (uint32_t)std::max<uint64_t>(1, (pairs + EQ_THREADS - 1) / EQ_THREADS);
  lg_intro_eq_kernel<false><<<blocks, EQ_THREADS, 0, s>>>(f, point, n_vars, nullptr, 0, nullptr, pairs, pend, part, pub);
  LAUNCH_OK();
}
void launch_lg_intro_eq(const F256d* f, const F128d* eq_lo, uint32_t lo_bits, const F128d* eq_hi, uint64_t pairs,
                        F128d* pend, F128d* part, cudaStream_t s, FusedPublish pub) {
  const uint32_t blocks =
      (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((pairs + EQ_THREADS - 1) / EQ_THREADS, (uint64_t)sm_count() * 8));
  lg_intro_eq_kernel<true><<<blocks, EQ_THREADS, 0, s>>>(f, nullptr, 0, eq_lo, lo_bits, eq_hi, pairs, pend, part, pub);
  LAUNCH_OK();
}
// Induced basis of the queried positions. The level's codeword is the NTT (layers
// [log_rate, log_d)) of the message replicated 2^log_rate times, so for weights w_q at
// positions pos_q
//   basis = R^T . L_rate^T ... L_{log_d-1}^T . (sum_q w_q e_{pos_q}),
// with the transposed butterfly (u, v) -> (u + v, v + t (u + v)) and R^T the sum over
// the replicas. One scatter, log_d - log_rate transposed layers and the replica fold.
__global__ void lg_scatter_kernel(const uint64_t* __restrict__ pos, const F128d* __restrict__ w, uint32_t n_q,
                                  F128d* __restrict__ y) {
  uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n_q) return;
  unsigned long long* p = reinterpret_cast<unsigned long long*>(y + pos[q]);
  atomicXor(p, (unsigned long long)w[q].lo);
  atomicXor(p + 1, (unsigned long long)w[q].hi);
}
__global__ void ntt_t_layer_kernel(F128d* __restrict__ y, uint32_t log_d, uint32_t layer, const F128d* __restrict__ tw) {
  uint64_t pair = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (pair >= (1ull << (log_d - 1))) return;
  uint32_t sh = log_d - layer - 1;
  uint64_t blk = pair >> sh, within = pair & ((1ull << sh) - 1);
  uint64_t i0 = (blk << (sh + 1)) + within, i1 = i0 + (1ull << sh);
  F128d t = tw[(1ull << layer) - 1 + blk];
  F128d u = y[i0], v = y[i1], sum = u + v;
  y[i0] = sum;
  y[i1] = blk == 0 ? v : v + t * sum;  // the first block's twiddle is zero in every layer
}
// basis[i] = sum_rep y[rep * n + i]; with the split f (length 2n):
// a = sum f[2i] basis[i], s = sum (f[2i] + f[2i+1]) basis[i].
__global__ void lg_induced_fold_kernel(const F128d* __restrict__ y, uint32_t ln, uint32_t log_rate,
                                       const F256d* __restrict__ f, F128d* __restrict__ basis, F128d* __restrict__ part,
                                       FusedPublish pub) {
  __shared__ F128d sh[32];
  uint64_t n = 1ull << ln;
  F128d A = f128_zero(), Sm = f128_zero();
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    F128d acc = f128_zero();
    for (uint64_t rep = 0; rep < (1ull << log_rate); ++rep) acc += y[rep * n + i];
    basis[i] = acc;
    F128d f0 = f[2 * i].c0, f1 = f[2 * i + 1].c0;
    A += f0 * acc;
    Sm += (f0 + f1) * acc;
  }
  A = block_xor(A, sh);
  Sm = block_xor(Sm, sh);
  if (threadIdx.x == 0) { part[blockIdx.x * 2] = A; part[blockIdx.x * 2 + 1] = Sm; }
  if (pub.out) publish_if_last(part, 2, pub, sh);
}
// Several consecutive transposed layers in one launch: layers layer_hi, layer_hi - 1, ...,
// layer_hi - nl + 1 (pair distances 2^sh_min, ..., 2^(sh_min + nl - 1), sh_min =
// log_d - 1 - layer_hi) act within groups of 2^nl positions spaced 2^sh_min apart, so one
// block stages a group in shared memory and runs all nl layers there (one launch and one
// global pass instead of nl). Group g: base = (g >> sh_min) << (sh_min + nl) | (g mod
// 2^sh_min); position t of the group is base + t 2^sh_min. The butterfly is ntt_t_layer's.
constexpr uint32_t NTT_T_FUSED = 6;  // layers per fused pass (64-position groups)
constexpr uint32_t NTT_T_FUSED_MAX_LOG = 16;  // transforms of at most 2^16 positions use it
__global__ void __launch_bounds__(256)
ntt_t_fused_kernel(F128d* __restrict__ y, uint32_t log_d, uint32_t layer_hi, uint32_t nl,
                   const F128d* __restrict__ tw) {
  __shared__ F128d g[4][1u << NTT_T_FUSED];  // four groups per 256-thread block
  const uint32_t P = 1u << nl, sh_min = log_d - 1 - layer_hi;
  const uint64_t n_groups = 1ull << (log_d - nl);
  const uint32_t sub = threadIdx.x >> 6, t = threadIdx.x & 63;  // 64 threads per group
  const uint64_t gi = (uint64_t)blockIdx.x * 4 + sub;
  const bool have = gi < n_groups;  // group-uniform
  const uint64_t base = have ? (((gi >> sh_min) << (sh_min + nl)) | (gi & ((1ull << sh_min) - 1))) : 0;
  if (have && t < P) g[sub][t] = y[base + ((uint64_t)t << sh_min)];
  __syncthreads();
  for (uint32_t k = 0; k < nl; ++k) {
    const uint32_t layer = layer_hi - k, sh = sh_min + k;
    if (have && t < P / 2) {
      // pair t of the group at group distance 2^k
      const uint32_t lo = ((t >> k) << (k + 1)) | (t & ((1u << k) - 1)), hi = lo + (1u << k);
      const uint64_t i0 = base + ((uint64_t)lo << sh_min);
      const uint64_t blk = i0 >> (sh + 1);
      const F128d u = g[sub][lo], v = g[sub][hi], sum = u + v;
      g[sub][lo] = sum;
      g[sub][hi] = blk == 0 ? v : v + mul_call(tw[(1ull << layer) - 1 + blk], sum);  // first block: twiddle zero
    }
    __syncthreads();
  }
  if (have && t < P) y[base + ((uint64_t)t << sh_min)] = g[sub][t];
}
// The first transposed layers of a large level act on a vector that is zero but for the queried
// positions: within the 2^L positions of a query's block they leave
//   w prod_{k in bits(i)} (t_k + bit_k(pos)),  t_k the twiddle of layer k at pos >> (k + 1),
// at position i, so those layers are formed directly (two products an entry and query, sixteen
// values per four layers in shared memory) for the blocks that hold queries, instead of L passes
// over the whole vector (Ligerito of Keccak-f 2^18 9.2 -> 8.4 ms, 35 launches fewer). Block (group of queries with one block, ENTRIES entries of it).
constexpr uint32_t SPARSE_ENTRIES = 1024, SPARSE_MAX_LAYERS = 12;
__global__ void __launch_bounds__(256)
ntt_t_sparse_kernel(const uint64_t* __restrict__ pos, const F128d* __restrict__ w, const uint32_t* __restrict__ start,
                    uint32_t log_d, uint32_t L, const F128d* __restrict__ tw, F128d* __restrict__ y) {
  __shared__ F128d fac[SPARSE_MAX_LAYERS];
  __shared__ F128d sub[SPARSE_MAX_LAYERS / 4][16];
  const uint32_t q0 = start[blockIdx.x], q1 = start[blockIdx.x + 1], n = 1u << L;
  F128d acc[SPARSE_ENTRIES / 256];
#pragma unroll
  for (uint32_t e = 0; e < SPARSE_ENTRIES / 256; ++e) acc[e] = f128_zero();
  for (uint32_t q = q0; q < q1; ++q) {
    const uint64_t p = pos[q];
    __syncthreads();  // the previous query's tables are no longer read
    if (threadIdx.x < SPARSE_MAX_LAYERS) {
      const uint32_t k = threadIdx.x;
      F128d f = f128_one();
      if (k < L) {
        f = tw[(1ull << (log_d - 1 - k)) - 1 + (p >> (k + 1))];
        f.lo ^= (p >> k) & 1;
      }
      fac[k] = f;
    }
    __syncthreads();
    if (threadIdx.x < SPARSE_MAX_LAYERS * 4) {
      const uint32_t g = threadIdx.x >> 4, v = threadIdx.x & 15;
      F128d f[4];
#pragma unroll
      for (uint32_t b = 0; b < 4; ++b) f[b] = (v >> b) & 1 ? fac[4 * g + b] : f128_one();
      F128d s = mul_call(mul_call(f[0], f[1]), mul_call(f[2], f[3]));
      if (g == 0) s = mul_call(s, w[q]);
      sub[g][v] = s;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t e = 0; e < SPARSE_ENTRIES / 256; ++e) {
      const uint32_t i = blockIdx.y * SPARSE_ENTRIES + e * 256 + threadIdx.x;
      acc[e] += mul_call(mul_call(sub[0][i & 15], sub[1][(i >> 4) & 15]), sub[2][(i >> 8) & 15]);
    }
  }
  const uint64_t base = (pos[q0] >> L) << L;
#pragma unroll
  for (uint32_t e = 0; e < SPARSE_ENTRIES / 256; ++e) {
    const uint32_t i = blockIdx.y * SPARSE_ENTRIES + e * 256 + threadIdx.x;
    if (i < n) y[base + i] = acc[e];
  }
}
// Layers formed that way: blocks of 2^(log_d - 9) positions, so that few of a level's queries (at
// most 279) share one; levels of at most 2^NTT_T_FUSED_MAX_LOG positions run fused instead.
uint32_t lg_sparse_layers(uint32_t log_d, uint32_t log_rate) {
  return log_d > NTT_T_FUSED_MAX_LOG ? std::min({SPARSE_MAX_LAYERS, log_d - 9, log_d - log_rate}) : 0;
}
uint32_t launch_lg_induced(const uint64_t* pos, const F128d* w, uint32_t n_q, const uint32_t* start, uint32_t n_groups,
                           uint32_t ln, uint32_t log_rate, const F128d* tw, const F256d* f, F128d* y, F128d* basis,
                           F128d* part, cudaStream_t s, FusedPublish pub) {
  const uint32_t log_d = ln + log_rate, sparse = lg_sparse_layers(log_d, log_rate);
  CUDA_OK(cudaMemsetAsync(y, 0, (sizeof(F128d)) << log_d, s));
  if (sparse) {
    const uint32_t chunks = std::max(1u, (1u << sparse) / SPARSE_ENTRIES);
    ntt_t_sparse_kernel<<<dim3(n_groups, chunks), 256, 0, s>>>(pos, w, start, log_d, sparse, tw, y);
  } else {
    lg_scatter_kernel<<<(n_q + 127) / 128, 128, 0, s>>>(pos, w, n_q, y);
  }
  LAUNCH_OK();
  uint64_t pairs = 1ull << (log_d - 1);
  // transposed layers from log_d - 1 - sparse down to log_rate: for the small levels
  // (launch-latency bound) up to NTT_T_FUSED per launch; the large ones one per launch (their
  // fused groups would be strided and half the threads idle in every layer: slower, measured)
  const uint32_t per_launch = log_d <= NTT_T_FUSED_MAX_LOG ? NTT_T_FUSED : 1;
  for (int layer = (int)(log_d - 1 - sparse); layer >= (int)log_rate;) {
    const uint32_t nl = std::min<uint32_t>(per_launch, (uint32_t)(layer - (int)log_rate + 1));
    if (nl >= 2) {
      const uint64_t n_groups_t = 1ull << (log_d - nl);
      ntt_t_fused_kernel<<<(unsigned)((n_groups_t + 3) / 4), 256, 0, s>>>(y, log_d, (uint32_t)layer, nl, tw);
    } else {
      ntt_t_layer_kernel<<<(unsigned)((pairs + 255) / 256), 256, 0, s>>>(y, log_d, (uint32_t)layer, tw);
    }
    LAUNCH_OK();
    layer -= (int)nl;
  }
  uint64_t n = 1ull << ln;
  uint32_t blocks = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, (uint64_t)sm_count() * 8));
  lg_induced_fold_kernel<<<blocks, 256, 0, s>>>(y, ln, log_rate, f, basis, part, pub);
  LAUNCH_OK();
  return blocks;
}
// Glue a pending basis of n values p into b:
//   eq mode      : b[2i].c0 += w0 p[i], b[2i+1].c0 += w1 p[i]
//   induced mode : b[2i].c0 += w0 p[i], b[2i+1].c1 += w0 p[i]  (u * base = (0, base))
__global__ void lg_glue_kernel(F256d* __restrict__ b, const F128d* __restrict__ p, F128d w0, F128d w1, uint64_t n,
                               int induced) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const F128d v = p[i], e = mul_call(w0, v);
  b[2 * i].c0 += e;
  if (induced) b[2 * i + 1].c1 += e;
  else b[2 * i + 1].c0 += mul_call(w1, v);
}
void launch_lg_glue(F256d* b, const F128d* p, F128d w0, F128d w1, uint64_t n, bool induced, cudaStream_t s) {
  lg_glue_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(b, p, w0, w1, n, induced ? 1 : 0);
  LAUNCH_OK();
}

}  // namespace gpu
}  // namespace flock
