// Commitment kernels: the lane-major codeword fill, the additive NTT over GF(2^128)
// (LCH novel basis, neighbours-last: at layer l pairs are 2^(log_d - l - 1) apart and
// share the twiddle of their block; crates/flock-core/src/ntt/additive_ntt_f128.rs:
// 627-648), Merkle trees over codeword rows (crates/flock-core/src/merkle.rs:593-620)
// and the row / capped-path gathers of Ligerito openings
// (crates/flock-core/src/pcs/ligerito.rs:4582-4610, merkle.rs:663-690).
//
// Layout: codewords are position-major SoA, data[pos * lanes + lane]; a Merkle leaf is
// one position's `lanes` words. Trees are flat: leaves [0, N), then each level, root last.
#include "kernels.h"
#include "reduce.cuh"
#include "sha256.cuh"
#include "wintable.cuh"
#include <atomic>

namespace flock {
namespace gpu {

// cw[(rep * D + p) * lanes + l] = q[l * D + p]: 2^(log_pos - log_dim) replicas of the
// transposed lane-major stack (the state after the first log_inv_rate NTT layers).
// Tiled through shared memory: a 32-position x 32-lane tile per block.
__global__ void fill_lane_major_kernel(const F128d* __restrict__ q, F128d* __restrict__ cw, uint32_t lanes,
                                       uint32_t log_dim, uint64_t n_pos) {
  __shared__ F128d tile[32][33];
  uint64_t p0 = (uint64_t)blockIdx.x * 32;
  uint32_t l0 = blockIdx.y * 32;
  uint64_t D = 1ull << log_dim;
  // read: lane-major, consecutive threads -> consecutive positions
  for (int ly = threadIdx.y; ly < 32; ly += blockDim.y) {
    uint32_t l = l0 + ly;
    uint64_t p = p0 + threadIdx.x;
    if (l < lanes && p < n_pos) tile[ly][threadIdx.x] = q[(uint64_t)l * D + (p & (D - 1))];
  }
  __syncthreads();
  // write: position-major, consecutive threads -> consecutive lanes
  for (int py = threadIdx.y; py < 32; py += blockDim.y) {
    uint64_t p = p0 + py;
    uint32_t l = l0 + threadIdx.x;
    if (l < lanes && p < n_pos) cw[p * lanes + l] = tile[threadIdx.x][py];
  }
}

void launch_fill_lane_major(const F128d* q, F128d* cw, uint32_t lanes, uint32_t log_dim, uint32_t log_pos,
                            cudaStream_t s) {
  uint64_t n_pos = 1ull << log_pos;
  dim3 grid((unsigned)((n_pos + 31) / 32), (lanes + 31) / 32), block(32, 8);
  fill_lane_major_kernel<<<grid, block, 0, s>>>(q, cw, lanes, log_dim, n_pos);
  LAUNCH_OK();
}

// Table layers: butterfly layers whose twiddle blocks are large. Each block of a launch
// handles a contiguous share of one twiddle block's butterflies (2^cpb_log launch blocks
// per twiddle block), builds that twiddle's byte tables once and takes half of its
// products from them (load/store pipe), the other half from split twiddles (multiply
// pipe). The butterflies of twiddle block b of a layer are the contiguous element ranges
// u = [b 2^(sh+1) lanes, + 2^sh lanes) and v = u + 2^sh lanes, sh = log_d - layer - 1
// (lane-minor layout); the first twiddle block's twiddle is zero in every layer.
//
// Two layers per pass, byte tables: twiddle block b of `layer` spans the quarters x0..x3 of
// Q = lanes 2^(sh-1) elements each; `layer` pairs (x0, x2) and (x1, x3) by t_b (table),
// layer + 1 pairs (x0, x1) by t_2b and (x2, x3) by t_2b+1 (split). One read and one write
// of the data per two layers.
__global__ void __launch_bounds__(256, 3)
ntt_layer2_tbl_kernel(F128d* __restrict__ data, uint32_t lanes, uint32_t log_d, uint32_t layer,
                      const F128d* __restrict__ tw, uint32_t cpb_log) {
  extern __shared__ __align__(16) F128d ttab[];  // build_byte_table's BYTE_TABLE_SMEM_ENTRIES
  __shared__ F128split s0, s1;
  const uint64_t b = blockIdx.x >> cpb_log, part = blockIdx.x & ((1ull << cpb_log) - 1);
  const uint32_t sh = log_d - layer - 1;
  const uint64_t Q = ((uint64_t)lanes) << (sh - 1);
  const uint64_t per = Q >> cpb_log;
  F128d* x = data + ((b << (sh + 1)) * lanes) + part * per;
  const bool zero = (b == 0);  // block-uniform: t_b and t_2b are zero
  if (threadIdx.x == 0) {
    s0 = split_factor(tw[(2ull << layer) - 1 + 2 * b]);
    s1 = split_factor(tw[(2ull << layer) - 1 + 2 * b + 1]);
  }
  if (!zero) build_byte_table(tw[(1ull << layer) - 1 + b], ttab);
  else __syncthreads();
  for (uint64_t k = threadIdx.x; k < per; k += blockDim.x) {
    F128d a0 = x[k], a1 = x[Q + k], a2 = x[2 * Q + k], a3 = x[3 * Q + k];
    if (!zero) {
      a0 += mul_table(a2, ttab);
      a1 += mul_table(a3, ttab);
    }
    a2 += a0;
    a3 += a1;
    if (!zero) a0 += mul_split(a1, s0);  // inline: 7-11 % faster than the out-of-line call here
    a1 += a0;
    a2 += mul_split(a3, s1);
    a3 += a2;
    x[k] = a0;
    x[Q + k] = a1;
    x[2 * Q + k] = a2;
    x[3 * Q + k] = a3;
  }
}
// The same from two window tables (wintable.cuh, five bits, 2 x 101 KB, one 512-thread block per
// SM): t_b and t_2b by table, t_2b+1 split, the next unit's elements loaded before this one's
// products. Per unit 9.75 cycles of the shared-memory pipe and one product of the multiply
// pipe. Keccak-f 2^18 (42 lanes, 2^22 positions): 1.86 ms a pass against 2.35 for the byte
// table, SHA-256 2^16 0.34 against 0.37. Its build is not hidden by other blocks, so the
// byte-table form (three blocks per SM) stays the better one where a twiddle serves few units:
// 5376 units 2.26 (byte) against 2.27 ms, 3200 units 0.373 against 0.399.
constexpr int NTT_WIN = 5;
constexpr uint32_t NTT_WIN_THREADS = 512;
__global__ void __launch_bounds__(NTT_WIN_THREADS, 1)
ntt_layer2_win_kernel(F128d* __restrict__ data, uint32_t lanes, uint32_t log_d, uint32_t layer,
                      const F128d* __restrict__ tw, uint32_t cpb_log) {
  extern __shared__ __align__(16) char wt[];  // t_b's table, then t_2b's
  __shared__ F128split s1;
  const uint64_t b = blockIdx.x >> cpb_log, part = blockIdx.x & ((1ull << cpb_log) - 1);
  const uint32_t sh = log_d - layer - 1, lane = win_lane();
  const uint64_t Q = ((uint64_t)lanes) << (sh - 1);
  const uint64_t per = Q >> cpb_log;
  F128d* x = data + ((b << (sh + 1)) * lanes) + part * per;
  const bool zero = (b == 0);  // block-uniform: t_b and t_2b are zero
  uint64_t k = threadIdx.x;
  F128d a0, a1, a2, a3;
  if (k < per) { a0 = x[k]; a1 = x[Q + k]; a2 = x[2 * Q + k]; a3 = x[3 * Q + k]; }
  if (threadIdx.x == 0) s1 = split_factor(tw[(2ull << layer) - 1 + 2 * b + 1]);
  if (!zero) {
    build_win_table<NTT_WIN>(tw[(1ull << layer) - 1 + b], wt);
    build_win_table<NTT_WIN>(tw[(2ull << layer) - 1 + 2 * b], wt + WinTable<NTT_WIN>::BYTES);
  }
  __syncthreads();
  for (; k < per; k += NTT_WIN_THREADS) {
    const uint64_t kn = k + NTT_WIN_THREADS;
    F128d n0, n1, n2, n3;
    if (kn < per) { n0 = x[kn]; n1 = x[Q + kn]; n2 = x[2 * Q + kn]; n3 = x[3 * Q + kn]; }
    if (!zero) {
      a0 += mul_win<NTT_WIN>(a2, wt, lane);
      a1 += mul_win<NTT_WIN>(a3, wt, lane);
    }
    a2 += a0;
    a3 += a1;
    if (!zero) a0 += mul_win<NTT_WIN>(a1, wt + WinTable<NTT_WIN>::BYTES, lane);
    a1 += a0;
    a2 += mul_split(a3, s1);
    a3 += a2;
    x[k] = a0;
    x[Q + k] = a1;
    x[2 * Q + k] = a2;
    x[3 * Q + k] = a3;
    a0 = n0; a1 = n1; a2 = n2; a3 = n3;
  }
}
// Two layers run as a table pass while the first one's twiddle blocks hold at least this many
// units (lanes 2^(sh-1)): from WIN units on with window tables, from TBL on with a byte table.
// Against fused passes down to the last layer: 42 lanes, 336 units 3.73 + 5.64 ms (three fused
// layers left) against 8.68 (five); 50 lanes, 800 units 0.436 + 1.08 (four left) against 1.62
// (six). Below TBL a pass is only taken while more than six layers are left, down to MORE units
// (13 lanes, 416 units: 0.074 + 0.203 against 0.38 ms for fused passes of four and three). Each launch block gets at least NTT_TBL_MIN_BLOCK_BUTTERFLIES of a twiddle block's
// butterflies, and the transform has to give every SM two such blocks.
constexpr uint64_t NTT_WIN_MIN_UNITS = 8192;
constexpr uint64_t NTT_TBL_MIN_UNITS = 768;
constexpr uint64_t NTT_TBL_MORE_UNITS = 256;
constexpr uint64_t NTT_TBL_MIN_BLOCK_BUTTERFLIES = uint64_t(1) << 12;

// Several consecutive layers [layer, layer + nl) fused through shared memory. A block
// owns 2^nl positions spaced 2^(log_d - layer - nl) apart (one residue class inside a
// block of the first fused layer) for a slice of lanes; each fused layer pairs positions
// within that set. Fused layer k meets 2^k twiddles; the block stages all 2^nl - 1 of them
// once, already split for mul_split, after the positions' data.
// BOTTOM >= 1 (the pass ends with the transform's last layer): with the basis x^i the twiddle of
// layer log_d - 1 - i is the i-th Carlitz polynomial of a polynomial a of degree below log_d, an
// integral one of degree (deg a - i) 2^i: below 32 for the last layer and below 64 for the one
// before (any log_d to 32), and for the third from last where log_d <= 18 (BOTTOM = 2), so their
// products take four and six of the nine partial ones. Five layers of 42 lanes and 2^22 positions:
// 10.6 ms with nine for all, 8.7 so.
constexpr uint32_t NTT_BOTTOM3_MAX_LOG = 18;
constexpr uint32_t NTT_MAX_THREADS = 320;  // with 3 blocks per SM: at most 64 registers a thread
template <int NL, int BOTTOM>
__global__ void __launch_bounds__(NTT_MAX_THREADS, 3)
ntt_fused_kernel(F128d* __restrict__ data, uint32_t lanes, uint32_t log_d, uint32_t layer, const F128d* __restrict__ tw,
                 uint32_t lane_tile) {
  extern __shared__ F128d sm[];  // [2^NL][lane_tile], then F128split[2^NL - 1]
  const uint32_t P = 1u << NL;
  F128split* tws = reinterpret_cast<F128split*>(sm + P * lane_tile);
  uint32_t stride_log = log_d - layer - NL;  // spacing of the positions in this group
  uint64_t n_groups = 1ull << (log_d - NL);
  uint64_t lane_tiles = (lanes + lane_tile - 1) / lane_tile;
  uint64_t gidx = blockIdx.x / lane_tiles;
  uint32_t lt = (uint32_t)(blockIdx.x % lane_tiles);
  if (gidx >= n_groups) return;
  // group -> (outer block of the first fused layer, residue within stride)
  uint64_t outer = gidx >> stride_log, resid = gidx & ((1ull << stride_log) - 1);
  uint64_t base = (outer << (stride_log + NL)) + resid;
  uint32_t l0 = lt * lane_tile;
  uint32_t nl_here = min(lane_tile, lanes - l0);
  // twiddle (k, blk) at tws[2^k - 1 + blk]: its global block at layer + k is (outer << k) + blk
  for (uint32_t t = threadIdx.x; t < P - 1; t += blockDim.x) {
    const uint32_t k = 31 - __clz(t + 1), blk = t + 1 - (1u << k);
    const F128d v = tw[(1ull << (layer + k)) - 1 + (outer << k) + blk];
    const uint64_t hl[3] = {v.lo, v.hi, v.lo ^ v.hi};
#pragma unroll
    for (int q = 0; q < 3; ++q) {  // split_factor(v), stored as it is formed
      const uint32_t y0 = (uint32_t)hl[q], y1 = (uint32_t)(hl[q] >> 32);
      split_classes(y0, tws[t].w[3 * q]);
      split_classes(y1, tws[t].w[3 * q + 1]);
      split_classes(y0 ^ y1, tws[t].w[3 * q + 2]);
    }
  }
  // (pair, lane) of this thread's first element or butterfly and the step between them
  const uint32_t pr0 = threadIdx.x / nl_here, ln0 = threadIdx.x - pr0 * nl_here;
  const uint32_t dpr = blockDim.x / nl_here, dln = blockDim.x - dpr * nl_here;
  auto step = [&](uint32_t& pr, uint32_t& l) {
    pr += dpr;
    l += dln;
    if (l >= nl_here) {
      l -= nl_here;
      ++pr;
    }
  };
  F128d* g = data + base * lanes + l0;
  const uint64_t g_stride = (uint64_t)lanes << stride_log;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NL; ++k) {  // the first layer reads global memory, the last one writes it
    const uint32_t half = P >> (k + 1);  // pairing distance inside the group (in group positions)
    uint32_t pr = pr0, l = ln0;
    for (uint32_t i = threadIdx.x; i < (P / 2) * nl_here; i += blockDim.x) {
      uint32_t blk = pr / half, w = pr - blk * half;
      uint32_t i0 = blk * 2 * half + w, i1 = i0 + half;
      F128d* pu = k == 0 ? g + i0 * g_stride + l : sm + i0 * lane_tile + l;
      F128d* pv = k == 0 ? g + i1 * g_stride + l : sm + i1 * lane_tile + l;
      F128d u = *pu, v = *pv;
      // the first block's twiddle is zero in every layer
      const F128split& t = tws[(1u << k) - 1 + blk];
      F128d nu = u;
      if (outer != 0 || blk != 0)
        nu += BOTTOM >= 1 && k == NL - 1 ? mul_split_deg32(v, t)
              : (BOTTOM >= 1 && k == NL - 2) || (BOTTOM >= 2 && k == NL - 3) ? mul_split_deg64(v, t)
                                                                             : mul_split(v, t);
      pu = k == NL - 1 ? g + i0 * g_stride + l : sm + i0 * lane_tile + l;
      pv = k == NL - 1 ? g + i1 * g_stride + l : sm + i1 * lane_tile + l;
      *pu = nu;
      *pv = v + nu;
      step(pr, l);
    }
    if (k < NL - 1) __syncthreads();
  }
}

// Threads per fused-NTT block for a lane tile: among the multiples of 32 in [192, 320], the
// one with the most busy resident warps per SM (resident warps, capped at 32, times the
// fraction of threads with a butterfly in a layer's passes). Cached per device and tile.
template <int NL, int BOTTOM>
static uint32_t ntt_block_threads(uint32_t lane_tile, size_t smem) {
  static std::atomic<uint32_t> cache[MAX_DEVICES][65];
  int dev = 0;
  CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= MAX_DEVICES || lane_tile > 64) throw std::runtime_error("fused NTT: bad device or lane tile");
  uint32_t best = cache[dev][lane_tile].load(std::memory_order_relaxed);
  if (best) return best;
  const uint32_t butterflies = (1u << (NL - 1)) * lane_tile;
  double best_score = -1.0;
  for (uint32_t t = 192; t <= NTT_MAX_THREADS; t += 32) {
    int blocks = 0;
    CUDA_OK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, ntt_fused_kernel<NL, BOTTOM>, (int)t, smem));
    const uint32_t passes = (butterflies + t - 1) / t;
    const double score = std::min(blocks * t / 32.0, 32.0) * butterflies / (double)(passes * t);
    if (score > best_score + 1e-9) {
      best_score = score;
      best = t;
    }
  }
  cache[dev][lane_tile].store(best, std::memory_order_relaxed);
  return best;
}

template <int NL, int BOTTOM>
static void launch_ntt_fused_pass(F128d* data, uint32_t lanes, uint32_t log_d, uint32_t layer, const F128d* tw,
                             cudaStream_t s) {
  const uint32_t lane_tile = lanes < 64 ? lanes : 64;
  const size_t tw_bytes = ((1u << NL) - 1) * sizeof(F128split);
  const uint64_t n_groups = 1ull << (log_d - NL), lane_tiles = (lanes + lane_tile - 1) / lane_tile;
  const size_t smem = (size_t)(1u << NL) * lane_tile * sizeof(F128d) + tw_bytes;
  set_dynamic_smem((const void*)ntt_fused_kernel<NL, BOTTOM>, (int)((1u << NL) * 64 * sizeof(F128d) + tw_bytes));
  const uint32_t threads = ntt_block_threads<NL, BOTTOM>(lane_tile, smem);
  ntt_fused_kernel<NL, BOTTOM><<<(unsigned)(n_groups * lane_tiles), threads, smem, s>>>(data, lanes, log_d, layer, tw, lane_tile);
  LAUNCH_OK();
}

template <int NL>
static void launch_ntt_fused(F128d* data, uint32_t lanes, uint32_t log_d, uint32_t layer, const F128d* tw,
                             cudaStream_t s) {
  if (layer + NL < log_d) launch_ntt_fused_pass<NL, 0>(data, lanes, log_d, layer, tw, s);
  else if (log_d > NTT_BOTTOM3_MAX_LOG) launch_ntt_fused_pass<NL, 1>(data, lanes, log_d, layer, tw, s);
  else launch_ntt_fused_pass<NL, 2>(data, lanes, log_d, layer, tw, s);
}

void launch_ntt(F128d* data, uint32_t lanes, uint32_t log_d, uint32_t start_layer, const F128d* tw, cudaStream_t s) {
  uint32_t layer = start_layer;
  // the top layers, whose twiddles are each shared by many butterflies: table passes
  const uint64_t butterflies = (uint64_t)lanes << (log_d - 1);
  const bool tables = butterflies >= (uint64_t)sm_count() * 2 * NTT_TBL_MIN_BLOCK_BUTTERFLIES;
  // launch blocks per twiddle block: about eight per SM in all, and each with at least
  // NTT_TBL_MIN_BLOCK_BUTTERFLIES of the `share` butterflies of its twiddle block
  auto blocks_log = [&](uint32_t l, uint64_t share, uint32_t max_log) {
    uint32_t c = 0;
    while (c < max_log && ((uint64_t)1 << (l + c + 1)) <= (uint64_t)sm_count() * 8 &&
           (share >> (c + 1)) >= NTT_TBL_MIN_BLOCK_BUTTERFLIES)
      ++c;
    return c;
  };
  constexpr uint32_t MAX_NL = 6;  // layers fused per pass
  while (tables && log_d - layer >= 3) {
    const uint32_t sh = log_d - layer - 1;
    const uint64_t units = (uint64_t)lanes << (sh - 1);
    if (units < (log_d - layer > MAX_NL ? NTT_TBL_MORE_UNITS : NTT_TBL_MIN_UNITS)) break;
    // a block's share counted in butterflies (two per unit and layer)
    const uint32_t c = blocks_log(layer, (uint64_t)lanes << sh, sh - 1);
    const unsigned blocks = (unsigned)(1ull << (layer + c));
    if (units >= NTT_WIN_MIN_UNITS) {
      const int smem = 2 * WinTable<NTT_WIN>::BYTES;
      set_dynamic_smem((const void*)ntt_layer2_win_kernel, smem);
      ntt_layer2_win_kernel<<<blocks, NTT_WIN_THREADS, smem, s>>>(data, lanes, log_d, layer, tw, c);
    } else {
      const int smem = (int)(BYTE_TABLE_SMEM_ENTRIES * sizeof(F128d));
      set_dynamic_smem((const void*)ntt_layer2_tbl_kernel, smem);
      ntt_layer2_tbl_kernel<<<blocks, 256, smem, s>>>(data, lanes, log_d, layer, tw, c);
    }
    LAUNCH_OK();
    layer += 2;
  }
  // the rest in as few fused passes as there can be, of even depth (nine layers: five and four)
  while (layer < log_d) {
    const uint32_t left = log_d - layer, passes = (left + MAX_NL - 1) / MAX_NL, nl = (left + passes - 1) / passes;
    switch (nl) {
      case 1: launch_ntt_fused<1>(data, lanes, log_d, layer, tw, s); break;
      case 2: launch_ntt_fused<2>(data, lanes, log_d, layer, tw, s); break;
      case 3: launch_ntt_fused<3>(data, lanes, log_d, layer, tw, s); break;
      case 4: launch_ntt_fused<4>(data, lanes, log_d, layer, tw, s); break;
      case 5: launch_ntt_fused<5>(data, lanes, log_d, layer, tw, s); break;
      default: launch_ntt_fused<6>(data, lanes, log_d, layer, tw, s); break;
    }
    layer += nl;
  }
}

// ---- Merkle
template <bool MULADD>
__global__ void merkle_leaves_kernel(const F128d* __restrict__ rows, uint32_t lanes, uint64_t n_leaves,
                                     uint32_t* __restrict__ tree) {
  uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n_leaves) return;
  // blocks of four 16-byte words, then the rest with the padding (80, zeros, the bit length)
  const uint4* w = reinterpret_cast<const uint4*>(rows + p * lanes);
  uint32_t st[8], m[16];
  sha256_init(st);
  auto put = [&](int i, uint4 v) {
    m[4 * i] = bswap32(v.x);
    m[4 * i + 1] = bswap32(v.y);
    m[4 * i + 2] = bswap32(v.z);
    m[4 * i + 3] = bswap32(v.w);
  };
  uint32_t b = 0;
  for (; b + 4 <= lanes; b += 4) {
#pragma unroll
    for (int i = 0; i < 4; ++i) put(i, __ldg(w + b + i));
    sha256_compress<MULADD>(st, m);
  }
#pragma unroll
  for (uint32_t i = 0; i < 4; ++i)
    put(i, b + i < lanes ? __ldg(w + b + i) : make_uint4(b + i == lanes ? 0x80u : 0u, 0, 0, 0));
  m[14] = 0;
  m[15] = lanes * 128;
  sha256_compress<MULADD>(st, m);
  uint4* o = reinterpret_cast<uint4*>(tree + p * 8);
  o[0] = make_uint4(bswap32(st[0]), bswap32(st[1]), bswap32(st[2]), bswap32(st[3]));
  o[1] = make_uint4(bswap32(st[4]), bswap32(st[5]), bswap32(st[6]), bswap32(st[7]));
}
__global__ void merkle_level_kernel(uint32_t* __restrict__ tree, uint64_t in_off, uint64_t n_out) {
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_out) return;
  const uint32_t* l = tree + (in_off + 2 * i) * 8;
  uint32_t out[8];
  sha256_words<true>([&](uint32_t k) { return l[k]; }, 16, out);
  uint64_t o = in_off + 2 * n_out + i;
#pragma unroll
  for (int k = 0; k < 8; ++k) tree[o * 8 + k] = out[k];
}
// Several small levels in one launch: a group of 2^(levels - 1) threads hashes 2^levels nodes up to
// one, a digest passing to the thread that needs it through shared memory. A level of few nodes
// is bound by the latency of its two compressions (about 5 us), whatever the launch; one block
// for all of them, which this replaced, was bound by its one SM (2048 nodes to 256: 28 us).
constexpr uint32_t MERKLE_SMALL_NODES = 1u << 15, MERKLE_SMALL_LEVELS = 3, MERKLE_SMALL_THREADS = 128;
__global__ void __launch_bounds__(MERKLE_SMALL_THREADS)
merkle_levels_kernel(uint32_t* __restrict__ tree, uint64_t in_off, uint64_t n_in, uint32_t levels,
                     uint32_t* __restrict__ cap, FusedPublish pub) {
  __shared__ uint32_t node[MERKLE_SMALL_THREADS][8];
  uint64_t off = in_off, len = n_in;
  const uint32_t t = threadIdx.x;
  uint32_t out[8];
  for (uint32_t k = 0; k < levels; ++k) {
    // thread t of the block holds node first + t of this level's output, the first ones only
    const uint32_t have = MERKLE_SMALL_THREADS >> k;
    const uint64_t nout = len / 2, i = (uint64_t)blockIdx.x * have + t;
    if (t < have && i < nout) {
      const uint32_t* l = tree + (off + 2 * i) * 8;
      sha256_words([&](uint32_t w) { return k ? node[2 * t + (w >> 3)][w & 7] : l[w]; }, 16, out);
#pragma unroll
      for (int w = 0; w < 8; ++w) tree[(off + len + i) * 8 + w] = out[w];
      if (cap && k == levels - 1) {
#pragma unroll
        for (int w = 0; w < 8; ++w) cap[i * 8 + w] = out[w];
      }
    }
    __syncthreads();  // this level's inputs are read
    if (t < have) {
#pragma unroll
      for (int w = 0; w < 8; ++w) node[t][w] = out[w];
    }
    __syncthreads();
    off += len;
    len = nout;
  }
  if (cap) publish_data(pub);
}
// The nodes [first, first + n) of the tree to mapped memory (a tree that is all cap).
__global__ void publish_nodes_kernel(const uint32_t* __restrict__ tree, uint32_t n, uint32_t* __restrict__ cap,
                                     FusedPublish pub) {
  for (uint32_t i = threadIdx.x; i < n * 8; i += blockDim.x) cap[i] = tree[i];
  publish_data(pub);
}
void launch_merkle(const F128d* rows, uint32_t lanes, uint64_t n_leaves, uint32_t cap_depth, uint8_t* tree,
                   cudaStream_t s, uint8_t* cap, FusedPublish pub) {
  // levels above the cap are never read (the cap is the commitment, paths stop below it)
  const uint64_t n_cap = uint64_t(1) << cap_depth;
  if (n_cap > n_leaves) throw std::runtime_error("Merkle cap wider than the leaf level");
  // from about a thousand leaves an SM on, the compressions are bound by the logic pipe, below
  // by their latency
  auto* leaves = n_leaves >= (uint64_t)sm_count() * 1024 ? merkle_leaves_kernel<true> : merkle_leaves_kernel<false>;
  leaves<<<(unsigned)((n_leaves + 127) / 128), 128, 0, s>>>(rows, lanes, n_leaves, (uint32_t*)tree);
  LAUNCH_OK();
  uint64_t off = 0, len = n_leaves;
  bool published = false;
  while (len > n_cap) {
    uint32_t levels = 1;
    if (len > MERKLE_SMALL_NODES) {
      merkle_level_kernel<<<(unsigned)((len / 2 + 127) / 128), 128, 0, s>>>((uint32_t*)tree, off, len / 2);
    } else {
      while (levels < MERKLE_SMALL_LEVELS && (len >> levels) > n_cap) ++levels;
      const bool last = (len >> levels) == n_cap;
      merkle_levels_kernel<<<(unsigned)((len / 2 + MERKLE_SMALL_THREADS - 1) / MERKLE_SMALL_THREADS), MERKLE_SMALL_THREADS, 0,
                             s>>>((uint32_t*)tree, off, len, levels, last ? (uint32_t*)cap : nullptr, pub);
      published |= last;
    }
    LAUNCH_OK();
    for (; levels; --levels) {
      off += len;
      len /= 2;
    }
  }
  if (cap && !published) {
    publish_nodes_kernel<<<1, 256, 0, s>>>((const uint32_t*)tree + off * 8, (uint32_t)n_cap, (uint32_t*)cap, pub);
    LAUNCH_OK();
  }
}

// ---- transcript proof of work (challenger.rs:1100-1140): the smallest nonce in
// [start, start + count) whose SHA256(digest || nonce_le) has `bits` leading zero bits,
// or ~0. Each block folds its minimum into *dmin; the last block to
// finish (ticket counter) reads and resets *dmin, writes the result to mapped host memory,
// then the sequence number, and resets the counter: one launch per search, no copies.
__global__ void __launch_bounds__(256) pow_kernel(uint4 dlo, uint4 dhi, uint32_t bits, uint64_t start, uint64_t count,
                                                  unsigned long long* dmin, uint32_t* counter, unsigned long long* out,
                                                  uint32_t* flag, uint32_t seq) {
  __shared__ unsigned long long bmin;
  __shared__ uint32_t ticket;
  if (threadIdx.x == 0) bmin = ~0ull;
  __syncthreads();
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) {
    const uint64_t nonce = start + i;
    uint32_t w[16];
    w[0] = bswap32(dlo.x); w[1] = bswap32(dlo.y); w[2] = bswap32(dlo.z); w[3] = bswap32(dlo.w);
    w[4] = bswap32(dhi.x); w[5] = bswap32(dhi.y); w[6] = bswap32(dhi.z); w[7] = bswap32(dhi.w);
    w[8] = bswap32((uint32_t)nonce);
    w[9] = bswap32((uint32_t)(nonce >> 32));
    w[10] = 0x80000000u;
#pragma unroll
    for (int k = 11; k < 15; ++k) w[k] = 0;
    w[15] = 320;
    uint32_t st[8];
    sha256_init(st);
    sha256_compress(st, w);
    bool ok = true;
    uint32_t need = bits;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (need >= 32) { ok &= st[k] == 0; need -= 32; }
      else if (need > 0) { ok &= (st[k] >> (32 - need)) == 0; need = 0; }
    }
    if (ok) atomicMin(&bmin, (unsigned long long)nonce);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (bmin != ~0ull) atomicMin(dmin, bmin);
    __threadfence();
    ticket = atomicAdd(counter, 1u);
  }
  __syncthreads();
  if (threadIdx.x == 0 && ticket == gridDim.x - 1) {
    __threadfence();
    const unsigned long long m = atomicExch(dmin, ~0ull);
    *counter = 0;
    *(volatile unsigned long long*)out = m;
    __threadfence_system();
    *(volatile uint32_t*)flag = seq;
  }
}
void launch_pow(const uint32_t digest_le[8], uint32_t bits, uint64_t start, uint64_t count, unsigned long long* d_min,
                uint32_t* d_counter, unsigned long long* out, uint32_t* flag, uint32_t seq, cudaStream_t s) {
  uint4 lo = make_uint4(digest_le[0], digest_le[1], digest_le[2], digest_le[3]);
  uint4 hi = make_uint4(digest_le[4], digest_le[5], digest_le[6], digest_le[7]);
  pow_kernel<<<(unsigned)((count + 255) / 256), 256, 0, s>>>(lo, hi, bits, start, count, d_min, d_counter, out, flag,
                                                             seq);
  LAUNCH_OK();
}

// ---- openings
// Rows and sibling paths of n positions straight to mapped memory, 16 bytes a thread: position q's
// row is `lanes` pieces, its path two per level (the sibling of pos >> k in level k, which starts
// at node 2 n_leaves - (2 n_leaves >> k)).
__global__ void gather_open_kernel(const uint4* __restrict__ mat, uint32_t lanes, const uint4* __restrict__ tree,
                                   uint64_t n_leaves, const uint64_t* __restrict__ pos, uint32_t n, uint32_t plen,
                                   uint4* __restrict__ rows, uint4* __restrict__ paths, FusedPublish pub) {
  const uint32_t per = lanes + 2 * plen, i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n * per) {
    const uint32_t q = i / per, r = i - q * per;
    if (r < lanes) {
      rows[q * lanes + r] = mat[pos[q] * lanes + r];
    } else {
      const uint32_t k = (r - lanes) >> 1, half = (r - lanes) & 1;
      const uint64_t node = 2 * n_leaves - ((2 * n_leaves) >> k) + ((pos[q] >> k) ^ 1);
      paths[(q * plen + k) * 2 + half] = tree[node * 2 + half];
    }
  }
  publish_data(pub);
}
void launch_gather_open(const F128d* mat, uint32_t lanes, const uint8_t* tree, uint64_t n_leaves, const uint64_t* d_pos,
                        uint32_t n, uint32_t cap_depth, F128d* rows, uint8_t* paths, cudaStream_t s, FusedPublish pub) {
  uint32_t depth = 0;
  while ((uint64_t(1) << depth) < n_leaves) ++depth;
  const uint32_t plen = depth - cap_depth, work = n * (lanes + 2 * plen);
  gather_open_kernel<<<std::max(1u, (work + 255) / 256), 256, 0, s>>>(
      reinterpret_cast<const uint4*>(mat), lanes, reinterpret_cast<const uint4*>(tree), n_leaves, d_pos, n, plen,
      reinterpret_cast<uint4*>(rows), reinterpret_cast<uint4*>(paths), pub);
  LAUNCH_OK();
}

}  // namespace gpu
}  // namespace flock
