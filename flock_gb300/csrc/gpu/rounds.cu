// The eq tables of many rounds in one launch, and the multipoint assist over a general jagged layout
// (union proofs): the dual values by the branching-program DP, and the two materialised vectors of
// its sumcheck with the first message; the rounds after it are pair_fold launches.
#include "assist.h"
#include "backend.h"
#include "reduce.cuh"

namespace flock {
namespace gpu {

// Several eq tables in one launch: table k = eq(point[off_k .. off_k + n_k)) at out +
// out_k. A block works on one table's entries [entry, entry + EQ_DESC_ENTRIES).
constexpr uint32_t EQ_DESC_ENTRIES = 1024;
__global__ void __launch_bounds__(EQ_THREADS)
eq_tables_kernel(const F128d* __restrict__ point, const EqDesc* __restrict__ desc, uint32_t n_desc,
                 F128d* __restrict__ out) {
  __shared__ F128d sub[EQ_MAX_GROUPS][16];
  uint32_t k = 0;
  uint64_t block = blockIdx.x;
  for (; k < n_desc; ++k) {  // the table of this block: tables take whole blocks, in order
    const uint64_t blocks = ((1ull << desc[k].n) + EQ_DESC_ENTRIES - 1) / EQ_DESC_ENTRIES;
    if (block < blocks) break;
    block -= blocks;
  }
  if (k == n_desc) return;
  const EqDesc d = desc[k];
  eq_sub_tables(point + d.p_off, d.n, sub);
  __syncthreads();
  const uint64_t end = min(uint64_t(1) << d.n, (block + 1) * EQ_DESC_ENTRIES);
  for (uint64_t i = block * EQ_DESC_ENTRIES + threadIdx.x; i < end; i += EQ_THREADS) out[d.out_off + i] = eq_from_sub(sub, d.n, i);
}
void launch_eq_tables(const F128d* point, const EqDesc* d_desc, const EqDesc* desc, uint32_t n_desc, F128d* out,
                      cudaStream_t s) {
  uint64_t blocks = 0;
  for (uint32_t k = 0; k < n_desc; ++k) blocks += ((1ull << desc[k].n) + EQ_DESC_ENTRIES - 1) / EQ_DESC_ENTRIES;
  eq_tables_kernel<<<(unsigned)blocks, EQ_THREADS, 0, s>>>(point, d_desc, n_desc, out);
  LAUNCH_OK();
}

// ------------------------------------------------------------------ the jagged multipoint assist
// Dual value ij = claim * n_points + j: sum over boundary runs of w * g_hat(z_row, point_j,
// t_c, t_next) by the width-4 branching program read from the top bit down
// (crates/flock-core/src/pcs/jagged.rs:164-192, 2547-2580). Block = one value, threads over
// runs. At a layer with bits (c, d) of the run's boundaries, state (carry, cmp) moves under
// (row, index = row + carry + c mod 2) to (carry' = (row + carry + c) / 2, cmp' = index == d ?
// cmp : d), so with V the states above and e[row + 2 index] the layer's eq weights
//   out[0][cmp] = e[0 + 2c] V[0][.] + e[1 + 2c'] V[c][.],
//   out[1][cmp] = e[0 + 2c'] V[c][.] + e[1 + 2c] V[1][.],   c' = 1 - c,
// where a factor V keeps cmp if its index equals d and has cmp = d otherwise: the terms that
// do not depend on cmp are formed once, six products a layer in both cases (c = d, c != d),
// selected without divergence. Bound by the multiply pipe (runs * layers * 6 products a
// value). With the whole assist on the host thread pool a three-type union of 2^13 rows
// (256 values, about 630 runs, 23 layers, 2^22 dense words) took 97.4 ms; with these kernels
// 12.9 ms, and a two-type one of 2^10 rows with 50 and 37 declared 10.4 -> 3.9 ms.
constexpr uint32_t DUAL_THREADS = 256;
constexpr uint32_t DUAL_MAX_LAYERS = 40;
__global__ void __launch_bounds__(DUAL_THREADS)
as_dual_kernel(const F128d* __restrict__ z_row, uint32_t n, const F128d* __restrict__ points, uint32_t m,
               uint32_t n_points, const ulonglong2* __restrict__ runs, const F128d* __restrict__ w, uint32_t n_runs,
               F128d* __restrict__ out) {
  __shared__ F128d e[DUAL_MAX_LAYERS * 4];
  __shared__ F128d sh[32];
  const uint32_t i = blockIdx.x / n_points, j = blockIdx.x % n_points, layers = m + 1;
  for (uint32_t q = threadIdx.x; q < layers * 4; q += blockDim.x) {
    const uint32_t l = q >> 2;
    F128d a = l < n ? z_row[i * n + l] : f128_zero(), b = l < m ? points[j * m + l] : f128_zero();
    if (!(q & 1)) a.lo ^= 1;  // 1 + a: row 0
    if (!(q & 2)) b.lo ^= 1;  // 1 + b: index 0
    e[q] = a * b;
  }
  __syncthreads();
  F128d acc = f128_zero();
  for (uint32_t r = threadIdx.x; r < n_runs; r += blockDim.x) {
    const ulonglong2 t = runs[r];
    // states v[carry][cmp]; the accepting state after the top layer is carry 0, cmp 1
    F128d v00 = f128_zero(), v01 = f128_one(), v10 = f128_zero(), v11 = f128_zero();
    for (int l = (int)layers - 1; l >= 0; --l) {
      const uint32_t c = (uint32_t)(t.x >> l) & 1, d = (uint32_t)(t.y >> l) & 1;
      const F128d* el = e + 4 * l;
      const F128d e0c = el[2 * c], e1c = el[1 + 2 * c], e0n = el[2 * (c ^ 1)], e1n = el[1 + 2 * (c ^ 1)];
      const F128d vc0 = c ? v10 : v00, vc1 = c ? v11 : v01;                                // V[c][.]
      const F128d v0d = d ? v01 : v00, v1d = d ? v11 : v10, vcd = d ? vc1 : vc0;            // cmp = d
      const bool same = c == d;
      const F128d X = same ? e0c : e1n, Y = same ? e1c : e0n, Z = same ? e1n : e0c, U = same ? e0n : e1c;
      const F128d p0 = mul_call(X, same ? v00 : vc0), p1 = mul_call(X, same ? v01 : vc1);
      const F128d p2 = mul_call(Y, same ? v10 : vc0), p3 = mul_call(Y, same ? v11 : vc1);
      const F128d p4 = mul_call(Z, same ? vcd : v0d), p5 = mul_call(U, same ? vcd : v1d);
      v00 = p0 + p4;
      v01 = p1 + p4;
      v10 = p2 + p5;
      v11 = p3 + p5;
    }
    acc += mul_call(w[i * n_runs + r], v00);
  }
  acc = block_xor(acc, sh);
  if (threadIdx.x == 0) out[blockIdx.x] = acc;
}
void launch_as_dual(const F128d* z_row, uint32_t n, const F128d* points, uint32_t m, uint32_t n_claims,
                    uint32_t n_points, const void* runs, const F128d* w, uint32_t n_runs, F128d* out, cudaStream_t s) {
  if (m + 1 > DUAL_MAX_LAYERS) throw std::runtime_error("assist: too many dense variables");
  as_dual_kernel<<<n_claims * n_points, DUAL_THREADS, 0, s>>>(z_row, n, points, m, n_points,
                                                              static_cast<const ulonglong2*>(runs), w, n_runs, out);
  LAUNCH_OK();
}

// abar[d] = er0[row] ec0[col] + er1[row] ec1[col] (zero past the area) and g[d] = T(eq(d)),
// T the GF(2)-linear map of the byte tables, with the first message over the pairs
// (2i, 2i + 1): g1 = sum abar[2i + 1] g[2i + 1], ginf = sum (abar[2i] + abar[2i + 1]) (g[2i] +
// g[2i + 1]). g is not zero past the area and enters later messages through pairs with one
// live entry, so the whole vectors are built and folded. One block of 512 threads per SM beside
// the 64 KB of tables; per entry three products and 16 lookups.
__global__ void __launch_bounds__(AS_BUILD_THREADS, 1)
as_build_kernel(const F128d* __restrict__ er0, const F128d* __restrict__ ec0, const F128d* __restrict__ er1,
                const F128d* __restrict__ ec1, const F128d* __restrict__ eq_lo, uint32_t lo_bits,
                const F128d* __restrict__ eq_hi, const F128d* __restrict__ table, uint64_t area, uint64_t n, JaggedSegs segs,
                F128d* __restrict__ abar, F128d* __restrict__ g, F128d* __restrict__ part, FusedPublish pub) {
  extern __shared__ __align__(16) F128d tab[];  // 16 x 256
  __shared__ F128d sh[32];
  for (uint32_t i = threadIdx.x; i < 16 * 256; i += blockDim.x) tab[i] = table[i];
  __syncthreads();
  F128d g1 = f128_zero(), gi = f128_zero();
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; 2 * i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    F128d A[2], G[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint64_t d = 2 * i + k;
      uint64_t row = 0, col = 0;
      A[k] = d < area && jagged_unrank(segs, d, row, col) ? mul_call(er0[row], ec0[col]) + mul_call(er1[row], ec1[col])
                                                          : f128_zero();
      G[k] = fold_slot(mul_call(eq_lo[d & ((1ull << lo_bits) - 1)], eq_hi[d >> lo_bits]), tab);
      abar[d] = A[k];
      g[d] = G[k];
    }
    g1 += mul_call(A[1], G[1]);
    gi += mul_call(A[0] + A[1], G[0] + G[1]);
  }
  g1 = block_xor(g1, sh);
  gi = block_xor(gi, sh);
  if (threadIdx.x == 0) { part[blockIdx.x * 2] = g1; part[blockIdx.x * 2 + 1] = gi; }
  publish_if_last(part, 2, pub, sh);
}
void launch_as_build(const F128d* er0, const F128d* ec0, const F128d* er1, const F128d* ec1, const F128d* eq_lo,
                     uint32_t lo_bits, const F128d* eq_hi, const F128d* table, uint64_t area, uint64_t n,
                     const JaggedSegs& segs, F128d* abar, F128d* g, F128d* part, cudaStream_t s, FusedPublish pub) {
  const int smem = 16 * 256 * (int)sizeof(F128d);
  set_dynamic_smem((const void*)as_build_kernel, smem);
  const uint32_t blocks = as_build_blocks(n, (uint64_t)sm_count());
  as_build_kernel<<<blocks, AS_BUILD_THREADS, smem, s>>>(er0, ec0, er1, ec1, eq_lo, lo_bits, eq_hi, table, area, n, segs, abar, g,
                                            part, pub);
  LAUNCH_OK();
}

// ------------------------------------------------------------------ host side
namespace {
inline F128d dev(F128 v) { return f128(v.lo, v.hi); }
constexpr uint32_t EQ_LO = 13;
}  // namespace

JaggedSegs jagged_segs(const Statement& S) {
  JaggedSegs g;
  uint64_t base = 0;
  for (const SlotInfo& T : S.slots) {
    if (!T.count || !T.used_cols) continue;
    if (g.n == 4) throw std::runtime_error("the merged weight supports at most four non-empty slots");
    g.base[g.n] = base;
    g.rows[g.n] = T.count;
    g.cols[g.n] = T.used_cols;
    g.col_off[g.n] = T.col_offset(S.nu);
    base += T.count * T.used_cols;
    g.n++;
  }
  return g;
}

template <class T>
T* JaggedAssist::alloc(size_t n) {
  void* p = nullptr;
  CUDA_OK(cudaMalloc(&p, std::max<size_t>(n, 1) * sizeof(T)));
  device_bytes_ += std::max<size_t>(n, 1) * sizeof(T);
  owned_.push_back(p);
  return static_cast<T*>(p);
}

// The largest call stages the points of 128 twists, every run and its weights.
static size_t assist_stage_bytes(const Statement& s) { return (size_t(1) << 18) + (size_t(48) << s.geo.col_log); }
constexpr uint32_t ASSIST_OUT = 256;  // dual values: two claims at 128 points

uint64_t JaggedAssist::estimate_device_bytes(const Statement& s, uint64_t sms) {
  const uint64_t n = s.committed_words;
  const uint32_t m = s.geo.dense_m - 7, lo = std::min(m, EQ_LO);
  uint64_t words = 0;
  for (int k = 0; k < 3; ++k) words += 2 * (n >> k);
  words += 2 * ((uint64_t(1) << s.nu) + (uint64_t(1) << s.geo.col_log)) + (uint64_t(1) << lo) + (uint64_t(1) << (m - lo));
  words += assist_partials(n, sms) + ASSIST_OUT;
  return words * sizeof(F128d) + sizeof(uint32_t) + assist_stage_bytes(s);
}

JaggedAssist::JaggedAssist(const Statement& s, int device) : S(s), device_(device) {
  CUDA_OK(cudaStreamCreateWithFlags(&st_, cudaStreamNonBlocking));
  n_ = S.committed_words;
  for (int k = 0; k < 3; ++k) {
    a_[k] = alloc<F128d>(n_ >> k);
    g_[k] = alloc<F128d>(n_ >> k);
  }
  const uint32_t m = S.geo.dense_m - 7, lo = std::min(m, EQ_LO);
  for (int i = 0; i < 2; ++i) {
    er_[i] = alloc<F128d>(size_t(1) << S.nu);
    ec_[i] = alloc<F128d>(size_t(1) << S.geo.col_log);
  }
  eq_lo_ = alloc<F128d>(size_t(1) << lo);
  eq_hi_ = alloc<F128d>(size_t(1) << (m - lo));
  part_ = alloc<F128d>(assist_partials(n_, (uint64_t)sm_count()));
  out_ = alloc<F128d>(ASSIST_OUT);
  counter_ = alloc<uint32_t>(1);
  CUDA_OK(cudaMemsetAsync(counter_, 0, sizeof(uint32_t), st_));
  stage_cap_ = assist_stage_bytes(S);
  d_stage_ = alloc<uint8_t>(stage_cap_);
  CUDA_OK(cudaMallocHost(&h_stage_, stage_cap_));
  CUDA_OK(cudaMallocHost(&h_out_, ASSIST_OUT * sizeof(F128d)));
  CUDA_OK(cudaHostAlloc(&h_pub_, 2 * sizeof(F128d), cudaHostAllocMapped));
  CUDA_OK(cudaHostGetDevicePointer(&d_pub_, h_pub_, 0));
  CUDA_OK(cudaHostAlloc(&h_flag_, 64, cudaHostAllocMapped));
  CUDA_OK(cudaHostGetDevicePointer(&d_flag_, h_flag_, 0));
  *(volatile uint32_t*)h_flag_ = 0;
  CUDA_OK(cudaStreamSynchronize(st_));
}

JaggedAssist::~JaggedAssist() {
  if (st_) cudaStreamSynchronize(st_);
  for (void* p : owned_) cudaFree(p);
  cudaFreeHost(h_stage_);
  cudaFreeHost(h_out_);
  cudaFreeHost(h_pub_);
  cudaFreeHost(h_flag_);
  if (st_) cudaStreamDestroy(st_);
}

// Every call waits for its own result, so staging starts over with each.
const void* JaggedAssist::upload(const void* src, size_t bytes) {
  const size_t off = (stage_off_ + 255) & ~size_t(255);
  if (off + bytes > stage_cap_) throw std::runtime_error("assist staging exhausted");
  memcpy(h_stage_ + off, src, bytes);
  CUDA_OK(cudaMemcpyAsync(d_stage_ + off, h_stage_ + off, bytes, cudaMemcpyHostToDevice, st_));
  stage_off_ = off + bytes;
  return d_stage_ + off;
}
FusedPublish JaggedAssist::publish() {
  FusedPublish p;
  p.out = d_pub_;
  p.flag = d_flag_;
  p.counter = counter_;
  p.seq = ++seq_;
  return p;
}
void JaggedAssist::read(const FusedPublish& p, bool stage, F128& g1, F128& gi) {
  GpuBackend::wait_flag(h_flag_, p.seq, st_, stage);
  const volatile F128d* o = h_pub_;
  g1 = F128(o[0].lo, o[0].hi);
  gi = F128(o[1].lo, o[1].hi);
}

void JaggedAssist::dual_values(const std::vector<AssistStatement>& unit, const std::vector<std::vector<F128>>& points,
                               uint32_t m, std::vector<std::vector<F128>>& values) {
  CUDA_OK(cudaSetDevice(device_));  // the assist's thread
  stage_off_ = 0;
  const size_t nc = unit.size(), np = points.size(), nr = unit[0].w.size(), n = unit[0].z_row.size();
  if (nc * np > ASSIST_OUT) throw std::runtime_error("assist: too many dual values");
  std::vector<F128> zr, pt, w;
  for (const AssistStatement& u : unit) {
    if (u.t != unit[0].t) throw std::runtime_error("assist: the claims' boundary runs differ");
    zr.insert(zr.end(), u.z_row.begin(), u.z_row.end());
    w.insert(w.end(), u.w.begin(), u.w.end());
  }
  for (const auto& p : points) pt.insert(pt.end(), p.begin(), p.end());
  std::vector<uint64_t> runs;
  for (const auto& t : unit[0].t) { runs.push_back(t.first); runs.push_back(t.second); }
  const auto* dz = static_cast<const F128d*>(upload(zr.data(), zr.size() * sizeof(F128)));
  const auto* dp = static_cast<const F128d*>(upload(pt.data(), pt.size() * sizeof(F128)));
  const auto* dw = static_cast<const F128d*>(upload(w.data(), w.size() * sizeof(F128)));
  const void* dr = upload(runs.data(), runs.size() * 8);
  launch_as_dual(dz, (uint32_t)n, dp, m, (uint32_t)nc, (uint32_t)np, dr, dw, (uint32_t)nr, out_, st_);
  CUDA_OK(cudaMemcpyAsync(h_out_, out_, nc * np * sizeof(F128d), cudaMemcpyDeviceToHost, st_));
  CUDA_OK(cudaStreamSynchronize(st_));
  for (size_t i = 0; i < nc; ++i)
    for (size_t j = 0; j < np; ++j) values[i][j] = F128(h_out_[i * np + j].lo, h_out_[i * np + j].hi);
}

void JaggedAssist::build(const std::vector<RsClaimPoint>& claims, const std::vector<F128>& scale,
                         const std::vector<F128>& rho, const std::vector<F128>& table, F128& g1, F128& gi) {
  CUDA_OK(cudaSetDevice(device_));
  stage_off_ = 0;
  if (claims.size() != 2) throw std::runtime_error("the assist expects the AB and C claims");
  for (int i = 0; i < 2; ++i) {
    std::vector<F128> rc(claims[i].z_row);
    rc.insert(rc.end(), claims[i].z_col.begin(), claims[i].z_col.end());
    const auto* p = static_cast<const F128d*>(upload(rc.data(), rc.size() * sizeof(F128)));
    launch_eq_split(p, (uint32_t)claims[i].z_row.size(), (uint32_t)claims[i].z_col.size(), dev(scale[i]), er_[i],
                    ec_[i], st_);
  }
  const uint32_t m = (uint32_t)rho.size(), lo = std::min(m, EQ_LO);
  const auto* pr = static_cast<const F128d*>(upload(rho.data(), rho.size() * sizeof(F128)));
  launch_eq_split(pr, lo, m - lo, f128_one(), eq_lo_, eq_hi_, st_);
  const auto* pt = static_cast<const F128d*>(upload(table.data(), table.size() * sizeof(F128)));
  FusedPublish fp = publish();
  launch_as_build(er_[0], ec_[0], er_[1], ec_[1], eq_lo_, lo, eq_hi_, pt, S.area(), n_, jagged_segs(S), a_[0], g_[0],
                  part_, st_, fp);
  cur_ = 0;
  len_ = n_;
  read(fp, true, g1, gi);
}

void JaggedAssist::fold(F128 r, F128& g1, F128& gi) {
  if (len_ < 4) throw std::runtime_error("assist: no fold left");
  const int nx = cur_ == 1 ? 2 : 1;
  const uint64_t n_pairs = len_ / 4;
  FusedPublish fp = publish();
  launch_pair_fold(a_[cur_], g_[cur_], n_pairs, n_pairs, dev(r), nullptr, 0, nullptr, nullptr, a_[nx], g_[nx], part_, st_,
                   fp);
  cur_ = nx;
  len_ /= 2;
  read(fp, false, g1, gi);
}

}  // namespace gpu
}  // namespace flock
