// The device backend of prove_fast: owns every witness-sized buffer in HBM for the
// life of a setup (z, a, b, the L0 codeword and tree, the zerocheck / merged-open fold
// buffers, the Ligerito F256 state and level codewords) and runs each bulk step of the
// protocol as sm_103a kernels on one stream. The host keeps only the transcript and the
// O(m)-sized arithmetic between rounds; every round message comes back as a handful of
// field elements.
#include "backend.h"
#include "wait.h"
#include "../host/tables.h"
#include <atomic>
#include <thread>

namespace flock {
namespace gpu {

namespace {

// Constant tables are per device (module constants and cudaMalloc'd tables live in each
// device's context); a process may drive several devices.
std::mutex g_consts_mu;
bool g_consts_done[MAX_DEVICES] = {};
void upload_constants_once() {
  int dev = 0;
  CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= MAX_DEVICES) throw std::runtime_error("device index out of range");
  std::lock_guard<std::mutex> g(g_consts_mu);
  if (g_consts_done[dev]) return;
  [] {
    const SkipTables& st = skip_tables();
    const uint8_t c[3] = {0xF7, 0x53, 0xB5};  // the three small zerocheck constants
    uint8_t e2[4];
    for (int K2 = 0; K2 < 4; ++K2) {
      uint8_t e = 1;
      for (int j = 0; j < 2; ++j) e = gf8_mul(e, ((K2 >> j) & 1) ? c[j + 1] : (uint8_t)(c[j + 1] ^ 1));
      e2[K2] = e;
    }
    // word 4M + K2 of an xo carries eq weight x^M * phi8(e2[K2]) (times D * eq_o(xo))
    F128 wconst[64], pconst[128];
    for (int M = 0; M < 16; ++M) {
      F128 xm = F128::one();
      for (int i = 0; i < M; ++i) xm = mul_by_x(xm);
      for (int K2 = 0; K2 < 4; ++K2) wconst[4 * M + K2] = xm * phi8(e2[K2]);
      for (int bit = 0; bit < 8; ++bit) pconst[8 * M + bit] = xm * phi8((uint8_t)(1u << bit));
    }
    std::vector<uint8_t> unit(64 * 64);
    for (int s = 0; s < 64; ++s)
      for (int i = 0; i < 64; ++i) unit[64 * s + i] = st.unit[s][i];
    upload_zc_consts(unit.data(), reinterpret_cast<const F128d*>(wconst), reinterpret_cast<const F128d*>(pconst));
    upload_witness_constants();
  }();
  g_consts_done[dev] = true;
}

inline F128d dev(F128 v) { F128d r; r.lo = v.lo; r.hi = v.hi; return r; }
inline F256d dev(F256 v) { F256d r; r.c0 = dev(v.c0); r.c1 = dev(v.c1); return r; }

}  // namespace

template <class T>
static T* dmalloc(size_t n, std::vector<void*>& owned, uint64_t& counter) {
  void* p = nullptr;
  if (n == 0) n = 1;
  CUDA_OK(cudaMalloc(&p, n * sizeof(T)));
  owned.push_back(p);
  counter += n * sizeof(T);
  return static_cast<T*>(p);
}

// The eq tables of the zerocheck, over coordinates [off, off + n) of the skip fold's point of
// length L: table 0 and 1 are the skip fold's low and high ones, tables 2 + 2i and 3 + 2i those
// of fold round i, whose message runs over the L - 1 - i coordinates from 1 + i on. Plain form
// (weighted = 0): each split as lo + hi, chunks of 2^8 pairs (one pair per thread). Weighted form
// with chunks of 2^w words: table 1 is the chunk weight h over [w, L), and the rounds i < w only
// have the low part [1 + i, w) of their coordinates.
struct ZcTable {
  uint32_t off, n;
};
static std::vector<ZcTable> zc_table_list(uint32_t L, uint32_t w) {
  std::vector<ZcTable> t;
  const uint32_t lo0 = w ? w : 10;
  t.push_back({0, lo0});
  t.push_back({lo0, L - lo0});
  for (uint32_t i = 0; i < L; ++i) {
    const uint32_t n = L - 1 - i;
    const uint32_t lo = i < w ? w - 1 - i : std::min(n, 8u);
    t.push_back({1 + i, lo});
    t.push_back({1 + i + lo, i < w ? 0 : n - lo});
  }
  return t;
}
static uint64_t zc_tables_entries(uint32_t L, uint32_t w) {
  uint64_t total = 0;
  for (const ZcTable& t : zc_table_list(L, w)) total += uint64_t(1) << t.n;
  return total;
}
// Words of z, a and b that can be nonzero: a single slot's witness fills chunk-columns
// c < used_cols of word (c << nu) + instance.
static uint64_t live_words_of(const Statement& S) {
  const uint64_t W = uint64_t(1) << (S.m - 7);
  return S.slots.size() == 1 && S.slots[0].offset == 0 ? std::min<uint64_t>(W, S.slots[0].used_cols << S.nu) : W;
}
// Room for either form (a degenerate challenge takes the plain one), and for the reciprocal
// weights beside the tables.
static uint64_t zc_tables_room(const Statement& S, uint64_t sms) {
  const uint32_t L = S.m - 7, w = zc_weighted_lo_bits(live_words_of(S), L, sms);
  return std::max(zc_tables_entries(L, 0), w ? zc_tables_entries(L, w) + (uint64_t(1) << (L - w)) : 0);
}

// Device bytes a backend for this statement holds after its first prove (the buffers of
// the constructor, the Ligerito level codewords and trees, the twiddle tables). Needs no device.
uint64_t GpuBackend::estimate_device_bytes(const Statement& S) {
  const uint64_t W = uint64_t(1) << (S.m - 7), K = uint64_t(1) << S.k_log, n_pos = uint64_t(1) << S.k_code;
  uint64_t b = 0;
  for (const SlotInfo& t : S.slots) b += t.count * input_record_bytes(t.hash);
  b += 3 * W * 16;                          // z, a, b
  if (!S.identity) b += S.committed_words * 16;  // the compacted stack
  b += n_pos * S.lanes * 16 + 2 * n_pos * 32;  // L0 codeword and tree
  b += (W / 2 * 2 + W * 2 + 64) * 16;       // zerocheck folds
  b += zc_tables_room(S, GB300_SMS) * 16;
  b += 6 * K * 16;                          // lincheck vectors
  for (const SlotInfo& t : S.slots) {
    b += 2 * (uint64_t(16) << t.k_log);
    if (t.csc_a)
      b += 4 * (t.csc_a->col_ptr.size() + t.csc_b->col_ptr.size()) + 2 * (t.csc_a->rows_flat.size() + t.csc_b->rows_flat.size());
  }
  b += (W + W + W / 2) * 16;                // merged weight and fold buffers
  const uint64_t D = uint64_t(1) << S.log_dim;
  b += lane_fold_groups(S.lanes, D, GB300_SMS) * D * 32;  // Ligerito: lane fold partials,
  b += 4 * 2 * D * 32 + 2 * D * 16;            // f/b ping-pong, pending
  b += uint64_t(PART_ENTRIES) * 16 + (size_t(96) << 20) + (size_t(8) << 20);  // partials, scratch, staging
  b += n_pos * 16;                          // L0 twiddles
  // recursive levels: codeword 2^(log_cols + rate) x 2^k, tree, twiddles
  const LigeritoParams& P = S.lig;
  uint32_t split_dim = (P.log_n - P.initial_k) + 1;
  for (uint32_t i = 0; i < P.r; ++i) {
    uint32_t k = P.recursive_ks[i], rate = P.log_inv_rates[i + 1];
    uint32_t log_cols = split_dim - k;
    uint64_t bl = uint64_t(1) << (log_cols + rate);
    b += bl * (uint64_t(1) << k) * 16 + 2 * bl * 32 + bl * 16;
    split_dim = (split_dim - k) + 1;
  }
  if (takes_jagged_assist(S)) b += JaggedAssist::estimate_device_bytes(S, GB300_SMS);
  return b;
}

GpuBackend::GpuBackend(const Statement& s) : S(s) {
  CUDA_OK(cudaGetDevice(&device_));
  CUDA_OK(cudaStreamCreateWithFlags(&st_, cudaStreamNonBlocking));
  upload_constants_once();
  W_ = uint64_t(1) << (S.m - 7);
  K_ = 1u << S.k_log;
  zc_live_words_ = live_words_of(S);
  const uint64_t W = W_;
  in_bytes_ = 0;
  for (const SlotInfo& t : S.slots) in_bytes_ += (size_t)t.count * input_record_bytes(t.hash);
  in_bytes_ = std::max<size_t>(in_bytes_, 16);
  d_in_ = dmalloc<uint8_t>(in_bytes_, owned_, device_bytes_);
  CUDA_OK(cudaMallocHost(&h_in_, in_bytes_));
  z_ = dmalloc<F128d>(W, owned_, device_bytes_);
  a_ = dmalloc<F128d>(W, owned_, device_bytes_);
  b_ = dmalloc<F128d>(W, owned_, device_bytes_);
  // chunk columns the witness never writes stay zero for the life of the backend
  CUDA_OK(cudaMemset(z_, 0, W * 16));
  CUDA_OK(cudaMemset(a_, 0, W * 16));
  CUDA_OK(cudaMemset(b_, 0, W * 16));
  n_pos0_ = uint64_t(1) << S.k_code;
  cw0_ = dmalloc<F128d>(n_pos0_ * S.lanes, owned_, device_bytes_);
  tree0_ = dmalloc<uint8_t>((2 * n_pos0_) * 32, owned_, device_bytes_);
  // fold buffers: round 2 writes W words per vector (zc2), later rounds alternate (zc1, zc2)
  zc1a_ = dmalloc<F128d>(W / 2, owned_, device_bytes_);
  zc1b_ = dmalloc<F128d>(W / 2, owned_, device_bytes_);
  zc2a_ = dmalloc<F128d>(W, owned_, device_bytes_);
  zc2b_ = dmalloc<F128d>(W, owned_, device_bytes_);
  zc_w64_ = dmalloc<F128d>(64 + 64 + 2 * 64, owned_, device_bytes_);  // weights, point, table list
  comb_ = dmalloc<F128d>(K_, owned_, device_bytes_);
  zv_ = dmalloc<F128d>(K_, owned_, device_bytes_);
  zvcap_ = dmalloc<F128d>(K_, owned_, device_bytes_);
  uint32_t k_max = 0;
  for (const SlotInfo& t : S.slots) {
    SlotDev sd;
    sd.K = 1u << t.k_log;
    k_max = std::max(k_max, sd.K);
    sd.ca = dmalloc<F128d>(sd.K, owned_, device_bytes_);
    sd.cb = dmalloc<F128d>(sd.K, owned_, device_bytes_);
    if (t.hash == HASH_KECCAK) {  // the walker writes the constrained columns only
      CUDA_OK(cudaMemsetAsync(sd.ca, 0, sd.K * 16, st_));
      CUDA_OK(cudaMemsetAsync(sd.cb, 0, sd.K * 16, st_));
    }
    if (t.hash != HASH_KECCAK) {
      for (auto [csc, d] : {std::make_pair(t.csc_a, &sd.a), std::make_pair(t.csc_b, &sd.b)}) {
        uint32_t* ptr = dmalloc<uint32_t>(csc->col_ptr.size(), owned_, device_bytes_);
        uint16_t* rows = dmalloc<uint16_t>(csc->rows_flat.size(), owned_, device_bytes_);
        CUDA_OK(cudaMemcpy(ptr, csc->col_ptr.data(), csc->col_ptr.size() * 4, cudaMemcpyHostToDevice));
        CUDA_OK(cudaMemcpy(rows, csc->rows_flat.data(), csc->rows_flat.size() * 2, cudaMemcpyHostToDevice));
        d->col_ptr = ptr;
        d->rows = rows;
      }
    }
    slot_dev_.push_back(sd);
  }
  eqi_ = dmalloc<F128d>(k_max, owned_, device_bytes_);
  ca_ = slot_dev_[0].ca;
  cb_ = slot_dev_[0].cb;
  Q_ = S.committed_words;
  q_ = S.identity ? z_ : dmalloc<F128d>(Q_, owned_, device_bytes_);
  mw_ = dmalloc<F128d>(W, owned_, device_bytes_);
  moAq_ = dmalloc<F128d>(W / 2, owned_, device_bytes_);
  moAw_ = dmalloc<F128d>(W / 2, owned_, device_bytes_);
  moBq_ = dmalloc<F128d>(W / 4, owned_, device_bytes_);
  moBw_ = dmalloc<F128d>(W / 4, owned_, device_bytes_);
  lane_part_ = dmalloc<F256d>(lane_fold_groups(S.lanes, rows(), (uint64_t)sm_count()) * rows(), owned_, device_bytes_);
  for (int k = 0; k < 2; ++k) {
    lf_[k] = dmalloc<F256d>(2 * rows(), owned_, device_bytes_);
    lb_[k] = dmalloc<F256d>(2 * rows(), owned_, device_bytes_);
  }
  pend_ = dmalloc<F128d>(2 * rows(), owned_, device_bytes_);
  static_assert(2 * TAIL >= 4 * LG_TAIL, "the tail buffer holds two F256 vectors of LG_TAIL entries");
  CUDA_OK(cudaHostAlloc(&h_tail_, 2 * TAIL * sizeof(F128d), cudaHostAllocMapped));
  CUDA_OK(cudaHostGetDevicePointer(&d_tail_, h_tail_, 0));
  part_cap_ = PART_ENTRIES;
  part_ = dmalloc<F128d>(part_cap_, owned_, device_bytes_);
  scr_cap_ = size_t(96) << 20;
  scr_ = dmalloc<uint8_t>(scr_cap_, owned_, device_bytes_);
  stage_cap_ = size_t(8) << 20;
  d_stage_ = dmalloc<uint8_t>(stage_cap_, owned_, device_bytes_);
  CUDA_OK(cudaMallocHost(&h_stage_, stage_cap_));
  CUDA_OK(cudaHostAlloc(&h_pub_, PUB_WORDS * sizeof(F128d), cudaHostAllocMapped));
  CUDA_OK(cudaHostGetDevicePointer(&d_pub_, h_pub_, 0));
  size_t open_bytes = 0;  // the largest opening: rows and whole paths of a level's queries
  for (uint32_t l = 0; l <= S.lig.r; ++l) {
    const size_t row = l ? size_t(16) << S.lig.recursive_ks[l - 1] : size_t(16) * S.lanes;
    open_bytes = std::max(open_bytes, S.lig.queries[l] * (row + 32 * 40));
  }
  d_open(open_bytes);
  CUDA_OK(cudaHostAlloc(&h_flag_, 64, cudaHostAllocMapped));
  CUDA_OK(cudaHostGetDevicePointer(&d_flag_, h_flag_, 0));
  *(volatile uint32_t*)h_flag_ = 0;
  pub_counter_ = dmalloc<uint32_t>(1, owned_, device_bytes_);
  CUDA_OK(cudaMemsetAsync(pub_counter_, 0, sizeof(uint32_t), st_));
  zc_tabs_cap_ = zc_tables_room(S, (uint64_t)sm_count());
  zc_tabs_ = dmalloc<F128d>(zc_tabs_cap_, owned_, device_bytes_);
  CUDA_OK(cudaStreamCreateWithFlags(&pow_st_, cudaStreamNonBlocking));
  d_pow_ = dmalloc<unsigned long long>(1, owned_, device_bytes_);
  CUDA_OK(cudaMemset(d_pow_, 0xFF, sizeof(unsigned long long)));
  pow_counter_ = dmalloc<uint32_t>(1, owned_, device_bytes_);
  CUDA_OK(cudaMemset(pow_counter_, 0, sizeof(uint32_t)));
  CUDA_OK(cudaHostAlloc(&h_pow_, sizeof(unsigned long long), cudaHostAllocMapped));
  CUDA_OK(cudaHostGetDevicePointer(&d_pow_out_, h_pow_, 0));
  CUDA_OK(cudaHostAlloc(&h_pow_flag_, 64, cudaHostAllocMapped));
  CUDA_OK(cudaHostGetDevicePointer(&d_pow_flag_, h_pow_flag_, 0));
  *(volatile uint32_t*)h_pow_flag_ = 0;
  // twiddles of the L0 transform; host tables used by every prove
  tw0_ = twiddles(S.k_code);
  (void)moore_inverse();
  if (takes_jagged_assist(S)) {
    jagged_ = std::make_unique<JaggedAssist>(S, device_);
    device_bytes_ += jagged_->device_bytes();
  }
  CUDA_OK(cudaDeviceSynchronize());
}

GpuBackend::~GpuBackend() {
  cudaStreamSynchronize(st_);
  for (void* p : owned_) cudaFree(p);
  for (auto& kv : tw_) cudaFree(kv.second);
  for (auto& L : levels_) { cudaFree(L.mat); cudaFree(L.tree); }
  for (cudaEvent_t e : ev_pool_) cudaEventDestroy(e);
  cudaFreeHost(h_in_);
  cudaFreeHost(h_open_);
  cudaFreeHost(h_stage_);
  cudaFreeHost(h_pow_);
  cudaFreeHost(h_pow_flag_);
  cudaFreeHost(h_pub_);
  cudaFreeHost(h_flag_);
  cudaFreeHost(h_tail_);
  cudaStreamDestroy(pow_st_);
  cudaStreamDestroy(st_);
}

const F128d* GpuBackend::twiddles(uint32_t log_d) {
  auto it = tw_.find(log_d);
  if (it != tw_.end()) return it->second;
  auto tw = ntt_twiddles(log_d);
  F128d* d = nullptr;
  CUDA_OK(cudaMalloc(&d, std::max<size_t>(1, tw.size()) * sizeof(F128d)));
  device_bytes_ += std::max<size_t>(1, tw.size()) * sizeof(F128d);
  // Ordered on this backend's stream: a plain cudaMemcpy from pageable memory may return
  // before its DMA lands, and kernels on a non-blocking stream are not ordered after it.
  CUDA_OK(cudaMemcpyAsync(d, tw.data(), tw.size() * sizeof(F128d), cudaMemcpyHostToDevice, st_));
  CUDA_OK(cudaStreamSynchronize(st_));
  tw_[log_d] = d;
  return d;
}

// ---- stage timing
const char* GpuBackend::stage_name(int s) {
  static const char* names[ST_COUNT] = {"witness", "l0_fill", "l0_ntt", "l0_merkle", "zc_round1", "zc_fold_skip",
                                        "zc_folds", "lincheck", "mo_build_w", "mo_rounds", "ligerito", "lg_ntt",
                                        "lg_merkle"};
  return (s >= 0 && s < ST_COUNT) ? names[s] : "?";
}
cudaEvent_t GpuBackend::event() {
  if (ev_used_ == ev_pool_.size()) {
    cudaEvent_t e;
    CUDA_OK(cudaEventCreate(&e));
    ev_pool_.push_back(e);
  }
  return ev_pool_[ev_used_++];
}
GpuBackend::Mark::Mark(GpuBackend* be, int stage) : b(be), st(stage), l0(launch_count()) {
  if ((b->timing_mask_ >> st) & 1) {
    cudaEvent_t a = b->event();
    CUDA_OK(cudaEventRecord(a, b->st_));
    b->spans_.push_back({st, a, nullptr, 0});
  }
}
GpuBackend::Mark::~Mark() {
  if (((b->timing_mask_ >> st) & 1) && !b->spans_.empty()) {
    cudaEvent_t e = b->event();
    if (cudaEventRecord(e, b->st_) == cudaSuccess) {
      b->spans_.back().b = e;
      b->spans_.back().launches = launch_count() - l0;
    }
  }
}
void GpuBackend::begin_prove(const void* d_inputs) {
  lg_pend_fold_.active = false;
  lg_pend_switch_ = false;
  lane_ = LaneStage();
  mo_lane_q_.clear();
  d_user_inputs_ = d_inputs;
  h2d_ = d2h_ = 0;
  spans_.clear();
  ev_used_ = 0;
}
void GpuBackend::stage_ms(double out[ST_COUNT], uint32_t launches[ST_COUNT]) {
  for (int i = 0; i < ST_COUNT; ++i) { out[i] = 0; launches[i] = 0; }
  CUDA_OK(cudaStreamSynchronize(st_));
  for (auto& sp : spans_) {
    if (!sp.b) continue;
    float ms = 0;
    CUDA_OK(cudaEventElapsedTime(&ms, sp.a, sp.b));
    out[sp.st] += ms;
    launches[sp.st] += (uint32_t)sp.launches;
  }
}

// ---- proof of work
uint64_t GpuBackend::gpu_pow(const std::array<uint8_t, 32>& digest, uint32_t bits) {
  std::lock_guard<std::mutex> g(pow_mu_);
  uint32_t words[8];
  memcpy(words, digest.data(), 32);
  // ~e^-16 chance that a window of 16 * 2^bits nonces holds no solution; then the next one
  const uint64_t window = uint64_t(16) << bits;
  for (uint64_t start = 0;; start += window) {
    const uint32_t seq = ++pow_seq_;
    launch_pow(words, bits, start, window, d_pow_, pow_counter_, d_pow_out_, d_pow_flag_, seq, pow_st_);
    wait_flag(h_pow_flag_, seq, pow_st_);
    const unsigned long long v = *(volatile unsigned long long*)h_pow_;
    if (v != ~0ull) return v;
  }
}
PowSearchFn GpuBackend::pow_search() {
  return [this](const std::array<uint8_t, 32>& digest, uint32_t bits) -> uint64_t {
    // Up to 8 bits (256 compressions expected) the host search with the SHA-2 instructions
    // (a few microseconds) beats a device launch and its round trip
    if (bits <= 8) return pow_search_host(digest, bits);
    return gpu_pow(digest, bits);
  };
}

// ---- staging helpers
void* GpuBackend::scratch(size_t bytes) {
  size_t off = (scr_off_ + 255) & ~size_t(255);
  if (off + bytes > scr_cap_) throw std::runtime_error("device scratch exhausted");
  scr_off_ = off + bytes;
  return scr_ + off;
}
const void* GpuBackend::upload(const void* src, size_t bytes) {
  size_t off = (stage_off_ + 255) & ~size_t(255);
  if (off + bytes > stage_cap_) {
    sync();
    off = 0;
  }
  memcpy(h_stage_ + off, src, bytes);
  CUDA_OK(cudaMemcpyAsync(d_stage_ + off, h_stage_ + off, bytes, cudaMemcpyHostToDevice, st_));
  h2d_ += bytes;
  stage_off_ = off + bytes;
  return d_stage_ + off;
}
void GpuBackend::upload_to(void* dst, const void* src, size_t bytes) {
  size_t off = (stage_off_ + 255) & ~size_t(255);
  if (off + bytes > stage_cap_) {
    sync();
    off = 0;
  }
  memcpy(h_stage_ + off, src, bytes);
  CUDA_OK(cudaMemcpyAsync(dst, h_stage_ + off, bytes, cudaMemcpyHostToDevice, st_));
  h2d_ += bytes;
  stage_off_ = off + bytes;
}
const F128d* GpuBackend::upload(const std::vector<F128>& v) {
  return static_cast<const F128d*>(upload(v.data(), v.size() * sizeof(F128)));
}
void GpuBackend::sync() {
  CUDA_OK(cudaStreamSynchronize(st_));
  stage_off_ = 0;
}
std::vector<F128> GpuBackend::reduce(uint32_t n_blocks, uint32_t width) {
  if ((uint64_t)n_blocks * width > part_cap_ || width > PUB_WORDS) throw std::runtime_error("partials buffer too small");
  const FusedPublish fp = fused_publish();
  launch_reduce_pair(part_, n_blocks, width, nullptr, 0, 0, st_, fp);
  return read_published(fp.seq, width);
}
std::vector<F128> GpuBackend::read_published(uint32_t seq, uint32_t width, bool stage) {
  wait_published(seq, stage);
  std::vector<F128> out(width);
  const volatile F128d* p = h_pub_;
  for (uint32_t j = 0; j < width; ++j) out[j] = F128(p[j].lo, p[j].hi);
  d2h_ += width * sizeof(F128d) + sizeof(uint32_t);
  return out;
}
// Wait for the published sequence number (the stream keeps running; no synchronisation).
void GpuBackend::wait_published(uint32_t seq, bool stage) { wait_flag(h_flag_, seq, st_, stage); }
void GpuBackend::wait_flag(const uint32_t* flag, uint32_t seq, cudaStream_t stream, bool stage) {
  wait_published_flag(flag, seq, stage, ROUND_WAIT_MS, [&] {
    const cudaError_t e = cudaStreamQuery(stream);
    if (e != cudaSuccess && e != cudaErrorNotReady) CUDA_OK(e);
    return e == cudaErrorNotReady;
  });
}
// eq(point) split as lo (first lo_bits coordinates) x hi (rest, times scale).
GpuBackend::EqSplit GpuBackend::eq_split(const std::vector<F128>& point, F128 scale, uint32_t max_lo) {
  EqSplit e;
  uint32_t n = (uint32_t)point.size();
  e.lo_bits = std::min(n, max_lo);
  uint32_t hi_bits = n - e.lo_bits;
  const F128d* dp = upload(point);
  F128d* lo = static_cast<F128d*>(scratch((size_t(16)) << e.lo_bits));
  F128d* hi = static_cast<F128d*>(scratch((size_t(16)) << hi_bits));
  launch_eq_split(dp, e.lo_bits, hi_bits, dev(scale), lo, hi, st_);
  e.lo = lo;
  e.hi = hi;
  return e;
}

// The eq tables over the coordinates [first, second) of args, in one launch; args (with anything else
// that the next kernel reads) travels in one copy, to the address returned.
const F128d* GpuBackend::eq_tables(std::vector<F128> args, const std::vector<std::pair<size_t, size_t>>& of,
                                   std::vector<F128d*>& out) {
  std::vector<EqDesc> desc(of.size());
  uint64_t total = 0;
  for (size_t k = 0; k < of.size(); ++k) {
    desc[k].p_off = (uint32_t)of[k].first;
    desc[k].n = (uint32_t)(of[k].second - of[k].first);
    desc[k].out_off = total;
    total += uint64_t(1) << desc[k].n;
  }
  F128d* tabs = static_cast<F128d*>(scratch(total * sizeof(F128d)));
  for (const EqDesc& d : desc) out.push_back(tabs + d.out_off);
  static_assert(sizeof(EqDesc) == sizeof(F128), "a descriptor takes the place of a word");
  const size_t words = args.size();
  args.resize(words + desc.size());
  memcpy(static_cast<void*>(args.data() + words), desc.data(), desc.size() * sizeof(EqDesc));
  const F128d* d = upload(args);
  launch_eq_tables(d, reinterpret_cast<const EqDesc*>(d + words), desc.data(), (uint32_t)desc.size(), tabs, st_);
  return d;
}

// ------------------------------------------------------------------ witness + commit
void GpuBackend::witness(const std::vector<const uint8_t*>& slot_inputs) {
  scr_off_ = 0;
  if (S.slots.size() != 1 || !S.identity) {
    // union: each slot's records are staged into consecutive regions of the input buffer;
    // the padded buffers are cleared (rows past a count, unused columns and gaps are zero)
    // and each slot's witness is written into its aligned block
    size_t off = 0;
    std::vector<size_t> offs;
    for (size_t t = 0; t < S.slots.size(); ++t) {
      const size_t bytes = (size_t)S.slots[t].count * input_record_bytes(S.slots[t].hash);
      offs.push_back(off);
      if (bytes) {
        memcpy(h_in_ + off, slot_inputs[t], bytes);
        CUDA_OK(cudaMemcpyAsync(d_in_ + off, h_in_ + off, bytes, cudaMemcpyHostToDevice, st_));
      }
      h2d_ += bytes;
      off += bytes;
    }
    Mark mk(this, ST_WITNESS);
    CUDA_OK(cudaMemsetAsync(z_, 0, W_ * 16, st_));
    CUDA_OK(cudaMemsetAsync(a_, 0, W_ * 16, st_));
    CUDA_OK(cudaMemsetAsync(b_, 0, W_ * 16, st_));
    for (size_t t = 0; t < S.slots.size(); ++t) {
      const SlotInfo& T = S.slots[t];
      if (!T.count) continue;
      const size_t w0 = T.offset >> 7;
      launch_witness((int)T.hash, d_in_ + offs[t], (uint32_t)T.count, S.nu, z_ + w0, a_ + w0, b_ + w0,
                     (uint32_t)T.used_cols, st_);
    }
    return;
  }
  const uint8_t* inputs = slot_inputs[0];
  const void* src = d_user_inputs_;
  if (!src) {
    // Host inputs: staged into pinned memory by the host thread pool, 8 MiB at a time, each
    // group's copy to the device queued as soon as it is staged (it overlaps the next
    // group's staging).
    const size_t GROUP = size_t(8) << 20, CHUNK = size_t(512) << 10;
    for (size_t g0 = 0; g0 < in_bytes_; g0 += GROUP) {
      const size_t glen = std::min(GROUP, in_bytes_ - g0);
      parallel_for((glen + CHUNK - 1) / CHUNK, [&](size_t c) {
        const size_t off = g0 + c * CHUNK;
        memcpy(h_in_ + off, inputs + off, std::min(CHUNK, g0 + glen - off));
      });
      CUDA_OK(cudaMemcpyAsync(d_in_ + g0, h_in_ + g0, glen, cudaMemcpyHostToDevice, st_));
    }
    h2d_ += in_bytes_;
    src = d_in_;
  }
  Mark mk(this, ST_WITNESS);
  launch_witness((int)S.hash, src, S.n_blocks, S.nu, z_, a_, b_, (uint32_t)S.geo.used_cols, st_);
}

void GpuBackend::commit_l0(uint32_t cap_depth, std::vector<Hash>& cap) {
  if (!S.identity) {
    // height-n_t compaction: each slot's used columns, the first `count` words of each,
    // stacked column after column (one strided copy per slot), then the zero tail
    Mark mk(this, ST_L0_FILL);
    uint64_t cursor = 0;
    for (const SlotInfo& T : S.slots) {
      if (!T.count || !T.used_cols) continue;
      CUDA_OK(cudaMemcpy2DAsync(q_ + cursor, T.count * 16, z_ + (T.offset >> 7), (size_t(16) << S.nu), T.count * 16,
                                T.used_cols, cudaMemcpyDeviceToDevice, st_));
      cursor += T.count * T.used_cols;
    }
    if (Q_ > cursor) CUDA_OK(cudaMemsetAsync(q_ + cursor, 0, (Q_ - cursor) * 16, st_));
  }
  { Mark mk(this, ST_L0_FILL); launch_fill_lane_major(q_, cw0_, S.lanes, S.log_dim, S.k_code, st_); }
  { Mark mk(this, ST_L0_NTT); launch_ntt(cw0_, S.lanes, S.k_code, 1, tw0_, st_); }
  const FusedPublish fp = fused_publish();
  {
    Mark mk(this, ST_L0_MERKLE);
    launch_merkle(cw0_, S.lanes, n_pos0_, cap_depth, tree0_, st_, d_open(size_t(32) << cap_depth), fp);
  }
  cap = read_cap(cap_depth, fp);
}

std::vector<Hash> GpuBackend::read_cap(uint32_t cap_depth, const FusedPublish& fp) {
  wait_published(fp.seq, true);
  std::vector<Hash> cap(size_t(1) << cap_depth);
  memcpy(cap.data(), h_open_, cap.size() * 32);
  d2h_ += cap.size() * 32;
  return cap;
}
// Mapped memory of at least `bytes` for a cap or an opening.
uint8_t* GpuBackend::d_open(size_t bytes) {
  if (bytes > open_cap_) {
    if (h_open_) {
      sync();
      cudaFreeHost(h_open_);
      h_open_ = nullptr;
      open_cap_ = 0;
    }
    CUDA_OK(cudaHostAlloc(&h_open_, bytes, cudaHostAllocMapped));
    CUDA_OK(cudaHostGetDevicePointer(&d_open_, h_open_, 0));
    open_cap_ = bytes;
  }
  return d_open_;
}

// ------------------------------------------------------------------ tails on the host
// Fold the low variable of both vectors at r; the message over the folded pairs, weighted by eq
// (empty: 1): g1 = sum eq A1 B1, ginf = sum eq (A0 + A1) (B0 + B1).
void GpuBackend::TailPair::fold(F128 r) {
  const size_t half = a.size() / 2;
  for (size_t i = 0; i < half; ++i) {
    a[i] = a[2 * i] + r * (a[2 * i + 1] + a[2 * i]);
    b[i] = b[2 * i] + r * (b[2 * i + 1] + b[2 * i]);
  }
  a.resize(half);
  b.resize(half);
}
void GpuBackend::TailPair::message(const std::vector<F128>& eq, F128& g1, F128& gi) const {
  g1 = gi = F128();
  for (size_t j = 0; 2 * j + 1 < a.size(); ++j) {
    const F128 t1 = a[2 * j + 1] * b[2 * j + 1], ti = (a[2 * j] + a[2 * j + 1]) * (b[2 * j] + b[2 * j + 1]);
    g1 += eq.empty() ? t1 : eq[j] * t1;
    gi += eq.empty() ? ti : eq[j] * ti;
  }
}
// The two vectors of n entries that a published one-block fold left in mapped memory.
GpuBackend::TailPair GpuBackend::read_tail(size_t n) {
  TailPair t;
  const volatile F128d* m = h_tail_;
  for (size_t i = 0; i < n; ++i) {
    t.a.push_back(F128(m[i].lo, m[i].hi));
    t.b.push_back(F128(m[n + i].lo, m[n + i].hi));
  }
  d2h_ += 2 * n * sizeof(F128d);
  return t;
}

// ------------------------------------------------------------------ zerocheck
void GpuBackend::zc_round1(const std::vector<F128>& r, std::vector<F128>& ab, std::vector<F128>& c,
                           std::vector<F128>& svc) {
  scr_off_ = 0;
  const uint32_t m = S.m;
  const auto& fixed = zc_fixed_challenges();
  for (int i = 0; i < 7; ++i)
    if (r[6 + i] != fixed[i]) throw std::runtime_error("zerocheck round 1 expects the fixed challenges at r[6..13)");
  std::vector<F128> outer(r.begin() + 13, r.end());
  EqSplit e = eq_split(outer, F128::one(), 10);
  uint32_t nrows = 0;
  F128d* part_svc = part_ + part_cap_ / 2;
  {
    Mark mk(this, ST_ZC_ROUND1);
    launch_zc_round1(a_, b_, z_, m, zc_live_words_, e.lo, e.lo_bits, e.hi, zc2a_, part_, part_svc, part_cap_ / 2,
                     &nrows, st_);
  }
  const FusedPublish fp = fused_publish();
  launch_reduce_pair(part_, nrows, 64, part_svc, nrows, 128, st_, fp);
  auto v = read_published(fp.seq, 192, true);
  // D = prod (1 + g_i)^-1 over the medium constants' g_i = x^1, x^2, x^4, x^8
  static const F128 D = [] {
    F128 d = F128::one();
    for (int e : {1, 2, 4, 8}) d = d * inv(F128::one() + F128(1ull << e, 0));
    return d;
  }();
  ab.assign(64, F128());
  svc.assign(128, F128());
  for (int i = 0; i < 64; ++i) ab[i] = D * v[i];
  for (int i = 0; i < 128; ++i) svc[i] = D * v[64 + i];
  // P_c(i) = sum_s phi8(unit_s(i)) * S_s with S_s = sum_x eq(x) bit_s(z_x); row x = 2w + h
  // splits eq(r[6..m], x) = eq(r_6, h) * eq(r[7..m], w), so S_s = (1 + r_6) svc[s] + r_6 svc[64 + s].
  // phi8 is additive: sum over the set bits b of unit_s(i) of phi8(2^b) * S_s.
  const SkipTables& st = skip_tables();
  F128 T[8][64];
  for (int s = 0; s < 64; ++s) {
    F128 Ss = (F128::one() + r[6]) * svc[s] + r[6] * svc[64 + s];
    for (int bit = 0; bit < 8; ++bit) T[bit][s] = phi8((uint8_t)(1u << bit)) * Ss;
  }
  c.assign(64, F128());
  for (int i = 0; i < 64; ++i) {
    F128 acc;
    for (int s = 0; s < 64; ++s) {
      uint8_t u = st.unit[s][i];
      while (u) {
        int bit = __builtin_ctz(u);
        acc += T[bit][s];
        u &= u - 1;
      }
    }
    c[i] = acc;
  }
}

void GpuBackend::zc_fold_skip(const std::vector<F128>& w, const std::vector<F128>& eq_point, F128& g1, F128& gi) {
  scr_off_ = 0;
  const uint32_t L = (uint32_t)eq_point.size();  // m - 7
  if (L < 10) throw std::runtime_error("zerocheck skip fold needs m >= 17");
  // the weighted form divides by the high coordinates' eq once: none may be 0 or 1
  zc_w_ = zc_weighted_lo_bits(zc_live_words_, L, (uint64_t)sm_count());
  for (uint32_t j = zc_w_; zc_w_ && j < L; ++j)
    if (eq_point[j].is_zero() || eq_point[j] == F128::one()) zc_w_ = 0;
  // Every later fold round i uses eq over the suffix eq_point[1 + i ..]: build all the
  // tables now, in one launch.
  zc_desc_.clear();
  uint64_t total = 0;
  for (const ZcTable& t : zc_table_list(L, zc_w_)) {
    EqDesc d;
    d.p_off = t.off;
    d.n = t.n;
    d.out_off = total;
    zc_desc_.push_back(d);
    total += uint64_t(1) << t.n;
  }
  zc_inv_ = zc_tabs_ + total;
  if (total + (zc_w_ ? uint64_t(1) << (L - zc_w_) : 0) > zc_tabs_cap_) throw std::runtime_error("zerocheck eq tables: size mismatch");
  // the weights, the point and the table list in one copy, to a place of their own (the first
  // fold reads the weights again)
  std::vector<uint8_t> args(64 * sizeof(F128) + L * sizeof(F128) + zc_desc_.size() * sizeof(EqDesc));
  memcpy(args.data(), w.data(), 64 * sizeof(F128));
  memcpy(args.data() + 64 * sizeof(F128), eq_point.data(), L * sizeof(F128));
  memcpy(args.data() + (64 + L) * sizeof(F128), zc_desc_.data(), zc_desc_.size() * sizeof(EqDesc));
  upload_to(zc_w64_, args.data(), args.size());
  const F128d *dw = zc_w64_, *dp = zc_w64_ + 64;
  const EqDesc* ddesc = reinterpret_cast<const EqDesc*>(zc_w64_ + 64 + L);
  const FusedPublish fp = fused_publish();
  {
    Mark mk(this, ST_ZC_FOLD_SKIP);
    launch_eq_tables(dp, ddesc, zc_desc_.data(), (uint32_t)zc_desc_.size(), zc_tabs_, st_);
    // words from zc_live_words_ on are zero and add nothing to the message
    const F128d* hi = zc_tabs_ + zc_desc_[1].out_off;
    if (zc_w_) launch_zc_fold_skip_weighted(a_, b_, dw, zc_live_words_, zc_w_, zc_tabs_, hi, part_, st_, fp);
    else launch_zc_fold_skip(a_, b_, dw, zc_live_words_, zc_tabs_, 10, hi, part_, st_, fp);
  }
  if (zc_w_) {
    // reciprocals of 1 + r_j and r_j (one inversion of their product), then of the weights h;
    // queued behind the skip fold
    std::vector<F128> f, pre;
    F128 p = F128::one();
    for (uint32_t j = zc_w_; j < L; ++j)
      for (F128 v : {F128::one() + eq_point[j], eq_point[j]}) {
        f.push_back(v);
        pre.push_back(p);
        p = p * v;
      }
    F128 q = inv(p);
    for (size_t i = f.size(); i-- > 0;) {
      const F128 v = f[i];
      f[i] = q * pre[i];
      q = q * v;
    }
    launch_factor_table(upload(f), L - zc_w_, zc_inv_, st_);
  }
  auto v = read_published(fp.seq, 2);
  g1 = v[0];
  gi = v[1];
  zc_tail_ = TailPair();
  zc_cur_a_ = nullptr;  // the skip-folded vectors live only implicitly (a, b bits and the weights)
  zc_cur_b_ = nullptr;
  zc_len_ = 2 * W_;
  zc_live_ = 2 * zc_live_words_;
  zc_round_ = 0;
}

void GpuBackend::zc_fold(F128 rho, const std::vector<F128>& eq_point, F128& g1, F128& gi) {
  uint64_t n_pairs = zc_len_ / 4;
  if ((uint64_t(1) << eq_point.size()) != n_pairs) throw std::runtime_error("zerocheck fold: eq size mismatch");
  size_t k = 2 + 2 * zc_round_;
  if (k + 1 >= zc_desc_.size() ||
      zc_desc_[k].n + (zc_round_ < zc_w_ ? zc_desc_[1].n : zc_desc_[k + 1].n) != eq_point.size())
    throw std::runtime_error("zerocheck fold: round tables out of step");
  if (!zc_tail_.a.empty()) {
    zc_tail_.fold(rho);
    zc_tail_.message(build_eq(eq_point), g1, gi);
    zc_len_ /= 2;
    zc_round_++;
    return;
  }
  const EqDesc& lo = zc_desc_[k];
  const EqDesc& hi = zc_desc_[k + 1];
  // pairs (4 entries in, 2 out) from live_pairs on read only the zero tail
  const uint64_t live_pairs = std::min<uint64_t>(n_pairs, (zc_live_ + 3) / 4);
  // round 0 writes W words per vector into zc2; later rounds alternate zc1 <-> zc2
  F128d* oa = (zc_round_ == 0 || zc_cur_a_ == zc1a_) ? zc2a_ : zc1a_;
  F128d* ob = (zc_round_ == 0 || zc_cur_a_ == zc1a_) ? zc2b_ : zc1b_;
  const bool tail = zc_round_ > 0 && 2 * n_pairs == TAIL;
  if (tail) {
    oa = d_tail_;
    ob = d_tail_ + TAIL;
  }
  const FusedPublish fp = fused_publish();
  {
    Mark mk(this, ST_ZC_FOLDS);
    const F128d* elo = zc_tabs_ + lo.out_off;
    const bool weighted = zc_round_ < zc_w_;  // the low coordinates of the weighted form
    const F128d* ehi = weighted ? nullptr : zc_tabs_ + hi.out_off;
    if (zc_round_ == 0 && weighted) {
      launch_zc_fold2_weighted(a_, b_, zc_w64_, dev(rho), n_pairs, live_pairs, zc_w_, elo, zc_tabs_ + zc_desc_[1].out_off,
                               oa, ob, part_, st_, fp);
    } else if (zc_round_ == 0) {
      F128d* tabs = static_cast<F128d*>(scratch(4096 * sizeof(F128d)));
      launch_zc_fold2(a_, b_, zc_w64_, dev(rho), tabs, n_pairs, live_pairs, elo, lo.n, ehi, oa, ob, part_, st_, fp);
    } else {
      // the first fold past the weighted rounds divides by h
      launch_pair_fold(zc_cur_a_, zc_cur_b_, n_pairs, live_pairs, dev(rho), elo, lo.n, ehi,
                       zc_w_ && zc_round_ == zc_w_ ? zc_inv_ : nullptr, oa, ob, part_, st_, fp);
    }
  }
  auto v = read_published(fp.seq, 2);
  g1 = v[0];
  gi = v[1];
  if (tail) zc_tail_ = read_tail(TAIL);
  zc_cur_a_ = oa;
  zc_cur_b_ = ob;
  zc_len_ /= 2;
  zc_live_ = std::min(zc_len_, 2 * live_pairs);
  zc_round_++;
}

void GpuBackend::zc_final(F128 rho, F128& ae, F128& be) {
  if (zc_len_ != 2 || zc_tail_.a.size() != 2) throw std::runtime_error("zerocheck final fold expects two values");
  zc_tail_.fold(rho);
  ae = zc_tail_.a[0];
  be = zc_tail_.b[0];
}

// ------------------------------------------------------------------ lincheck
void GpuBackend::lc_comb(const std::vector<F128>& skip_w, const std::vector<F128>& xir) {
  scr_off_ = 0;
  for (size_t t = 0; t < S.slots.size(); ++t) {
    // slot t folds its own matrices by skip_w (x) eq(xir[.. k_log_t - 6])
    const SlotInfo& T = S.slots[t];
    const SlotDev& sd = slot_dev_[t];
    std::vector<F128> args(skip_w);  // 64 weights, then the eq table
    const std::vector<F128> er = build_eq(std::vector<F128>(xir.begin(), xir.begin() + (T.k_log - 6)));
    args.insert(args.end(), er.begin(), er.end());
    const F128d* dw = upload(args);
    Mark mk(this, ST_LINCHECK);
    launch_lc_eq_inner(dw, dw + 64, sd.K, eqi_, st_);
    lc_fold_slot(T.hash, sd);
  }
}

void GpuBackend::lc_fold_slot(HashKind hash, const SlotDev& sd) {
  if (hash == HASH_KECCAK) {
    // the walker's column folds on the device (no materialised matrices)
    static const KeccakColumnConsts kc = [] {
      KeccakColumnConsts c{};
      for (int r = 0; r < 24; ++r) c.rc[r] = kr1cs::RC[r];
      for (int a = 0; a < 5; ++a)
        for (int b = 0; b < 5; ++b) c.rho[a + 5 * b] = (uint8_t)(kr1cs::RHO[a][b] % 64);
      return c;
    }();
    launch_keccak_lincheck_columns(eqi_, sd.ca, sd.cb, kc, st_);
    return;
  }
  launch_csc_fold(sd.a, sd.b, sd.K, eqi_, sd.ca, sd.cb, st_);
}

void GpuBackend::lc_zvec(const std::vector<F128>& x_outer) {
  scr_off_ = 0;
  const uint32_t nu = S.nu;
  Mark mk(this, ST_LINCHECK);
  const EqSplit e = eq_split(x_outer, F128::one(), 10);
  // a single slot folds its used columns only; a union folds every union column (the
  // gaps and unused columns of z are zero)
  uint32_t used = S.slots.size() == 1 ? (uint32_t)S.slots[0].used_cols : K_ / 128;
  launch_lc_zvec(z_, nu, used, e.lo, e.lo_bits, e.hi, part_, part_cap_, K_, zv_, zvcap_, st_);
  lc_len_ = K_;
  lc_tail_ = TailPair();
}

void GpuBackend::lc_start(F128 alpha, const std::vector<SlotComb>& sc, F128& e1, F128& ei) {
  const FusedPublish fp = fused_publish();
  if (S.slots.size() == 1 && sc[0].offset == 0 && sc[0].weight == F128::one()) {
    Mark mk(this, ST_LINCHECK);
    launch_lc_start(ca_, cb_, dev(alpha), dev(sc[0].beta), sc[0].pin, K_, comb_, zv_, part_, st_, fp);
  } else {
    Mark mk(this, ST_LINCHECK);
    CUDA_OK(cudaMemsetAsync(comb_, 0, size_t(K_) * 16, st_));
    for (size_t t = 0; t < S.slots.size(); ++t)
      launch_lc_slot_comb(slot_dev_[t].ca, slot_dev_[t].cb, dev(alpha), dev(sc[t].weight), dev(sc[t].beta), sc[t].pin,
                          slot_dev_[t].K, comb_ + sc[t].offset, st_);
    launch_lc_top_message(comb_, zv_, K_, part_, st_, fp);
  }
  auto v = read_published(fp.seq, 2);
  e1 = v[0];
  ei = v[1];
}

void GpuBackend::lc_round(F128 r, bool last, F128& e1, F128& ei) {
  if (!lc_tail_.a.empty()) {  // the top variable of comb and zv, on the host
    std::vector<F128>&c = lc_tail_.a, &z = lc_tail_.b;
    const size_t h = c.size() / 2, q = h / 2;
    for (size_t i = 0; i < h; ++i) {
      c[i] = c[i] + r * (c[i + h] + c[i]);
      z[i] = z[i] + r * (z[i + h] + z[i]);
    }
    c.resize(h);
    z.resize(h);
    lc_len_ /= 2;
    e1 = ei = F128();
    for (size_t i = 0; i < q && !last; ++i) {
      e1 += c[i + q] * z[i + q];
      ei += (c[i] + c[i + q]) * (z[i] + z[i + q]);
    }
    return;
  }
  const bool tail = lc_len_ / 2 == TAIL;
  F128d* co = tail ? d_tail_ : comb_;
  F128d* zo = tail ? d_tail_ + TAIL : zv_;
  FusedPublish fp = fused_publish();
  { Mark mk(this, ST_LINCHECK); launch_lc_round(comb_, zv_, lc_len_, dev(r), co, zo, part_, st_, fp); }
  lc_len_ /= 2;
  auto v = read_published(fp.seq, 2);
  e1 = v[0];
  ei = v[1];
  if (tail) lc_tail_ = read_tail(TAIL);
}

void GpuBackend::lc_partial(std::vector<F128>& zp) {
  if (lc_len_ != 64 || lc_tail_.b.size() != 64) throw std::runtime_error("lincheck partial expects 64 values");
  zp = lc_tail_.b;
}

void GpuBackend::lc_matrix_evals(const std::vector<F128>& rest, const std::vector<F128>& zp,
                                 std::vector<Pair128>& evals) {
  for (size_t t = 0; t < S.slots.size(); ++t) {
    scr_off_ = 0;
    const SlotInfo& T = S.slots[t];
    std::vector<F128> args(zp);  // 64 partial values, then the eq table
    const std::vector<F128> er = build_eq(std::vector<F128>(rest.begin(), rest.begin() + (T.k_log - 6)));
    args.insert(args.end(), er.begin(), er.end());
    const F128d* dzp = upload(args);
    const F128d* der = dzp + 64;
    const FusedPublish fp = fused_publish();
    {
      Mark mk(this, ST_LINCHECK);
      launch_lc_matrix_evals(slot_dev_[t].ca, slot_dev_[t].cb, der, dzp, slot_dev_[t].K, part_, st_, fp);
    }
    auto v = read_published(fp.seq, 2);
    evals.push_back({v[0], v[1]});
  }
}

void GpuBackend::lc_s_hat_v(const std::vector<F128>& tail, std::vector<F128>& out) {
  auto et = build_eq(tail);
  const F128d* det = upload(et);
  const FusedPublish fp = fused_publish();
  { Mark mk(this, ST_LINCHECK); launch_lc_s_hat_v(zvcap_, det, (uint32_t)et.size(), st_, fp); }
  out = read_published(fp.seq, 128, true);
}

// ------------------------------------------------------------------ merged open
void GpuBackend::launch_build_w(const std::vector<WeightClaim>& cl, uint32_t nu, uint64_t area, const FusedPublish& fp) {
  if (cl.size() != 2) throw std::runtime_error("merged open expects the AB and C claims");
  // both claims' byte tables, then their points z_row and z_col
  std::vector<F128> args;
  std::vector<std::pair<size_t, size_t>> of;
  for (int i = 0; i < 2; ++i) args.insert(args.end(), cl[i].table.begin(), cl[i].table.end());
  for (int i = 0; i < 2; ++i)
    for (const std::vector<F128>* p : {&cl[i].z_row, &cl[i].z_col}) {
      of.emplace_back(args.size(), args.size() + p->size());
      args.insert(args.end(), p->begin(), p->end());
    }
  std::vector<F128d*> eq;
  const F128d* dt = eq_tables(std::move(args), of, eq);
  F128d *er[2] = {eq[0], eq[2]}, *ec[2] = {eq[1], eq[3]};
  if (S.slots.size() == 1 && S.identity) {
    launch_mo_build_w(q_, er[0], ec[0], er[1], ec[1], dt, nu, area, Q_, mw_, part_, st_, fp);
    return;
  }
  const JaggedSegs g = jagged_segs(S);
  launch_mo_build_w(q_, er[0], ec[0], er[1], ec[1], dt, nu, area, Q_, mw_, part_, st_, fp, &g);
}

void GpuBackend::mo_build_w(const std::vector<WeightClaim>& cl, uint32_t nu, uint64_t area, F128& u0, F128& u2) {
  scr_off_ = 0;
  const FusedPublish fp = fused_publish();
  {
    Mark mk(this, ST_MO_BUILD_W);
    launch_build_w(cl, nu, area, fp);
  }
  auto v = read_published(fp.seq, 2);
  u0 = v[0];
  u2 = v[1];
  mo_q_ = q_;
  mo_w_ = mw_;
  mo_len_ = Q_;
  mo_live_ = std::min<uint64_t>(Q_, area);
  mo_chal_.clear();
  mo_tail_ = TailPair();
  mo_lane_q_.clear();
}

void GpuBackend::mo_round(F128 r, bool last, F128& g1, F128& gi) {
  mo_chal_.push_back(r);
  if (!mo_tail_.a.empty()) {
    mo_tail_.fold(r);
    if (!last) mo_tail_.message({}, g1, gi);
    if (mo_tail_.a.size() == lanes_pow2()) mo_lane_q_ = mo_tail_.a;
    return;
  }
  F128d* oq = (mo_q_ == moAq_) ? moBq_ : moAq_;
  F128d* ow = (mo_q_ == moAq_) ? moBw_ : moAw_;
  uint64_t n_pairs = mo_len_ / 4;
  const uint64_t live_pairs = std::min<uint64_t>(n_pairs, (mo_live_ + 3) / 4);
  const bool tail = 2 * n_pairs == TAIL;
  if (tail) {
    oq = d_tail_;
    ow = d_tail_ + TAIL;
  }
  FusedPublish fp = fused_publish();
  {
    Mark mk(this, ST_MO_ROUNDS);
    launch_pair_fold(mo_q_, mo_w_, n_pairs, live_pairs, dev(r), nullptr, 0, nullptr, nullptr, oq, ow, part_, st_, fp);
  }
  mo_q_ = oq;
  mo_w_ = ow;
  mo_len_ /= 2;
  mo_live_ = std::min(mo_len_, 2 * live_pairs);
  auto v = read_published(fp.seq, 2);
  g1 = v[0];
  gi = v[1];
  if (tail) mo_tail_ = read_tail(TAIL);
}

F128 GpuBackend::mo_q_eval() {
  if (mo_tail_.a.size() != 1) throw std::runtime_error("merged open: the claim is evaluated after its last round");
  return mo_tail_.a[0];
}

// ------------------------------------------------------------------ Ligerito
// Lane dots h[l] = sum_p q[l D + p] eq(point[.. log_dim), p). The merged open folded q at its
// round challenges: the lane dots at that point are its last row fold.
std::vector<F128> GpuBackend::lane_dots(const std::vector<F128>& point) {
  if (!mo_lane_q_.empty() && mo_chal_.size() >= S.log_dim && point.size() >= S.log_dim &&
      std::equal(point.begin(), point.begin() + S.log_dim, mo_chal_.begin()))
    return mo_lane_q_;
  scr_off_ = 0;
  EqSplit e = eq_split(std::vector<F128>(point.begin(), point.begin() + S.log_dim), F128::one(), 10);
  uint32_t nb;
  { Mark mk(this, ST_LIGERITO); nb = launch_lg_lane_dots(q_, S.lanes, S.log_dim, e.lo, e.lo_bits, e.hi, part_, part_cap_, st_); }
  std::vector<F128> h = reduce(nb, S.lanes);
  h.resize(lanes_pow2());  // the lanes past the committed ones are zero
  return h;
}

void GpuBackend::add_lane_term(F128 coef, const std::vector<F128>& point) {
  LaneTerm t;
  t.coef = coef;
  t.row_point.assign(point.begin(), point.begin() + S.log_dim);
  for (F128 v : build_eq(std::vector<F128>(point.begin() + S.log_dim, point.end()))) t.e.push_back(F256(v));
  for (F128 v : (point == lane_.dot_point ? lane_.dots : lane_dots(point))) t.h.push_back(F256(v));
  if (lane_.terms.size() == LaneTerms::MAX) throw std::runtime_error("too many basis terms");
  lane_.terms.push_back(std::move(t));
}

void GpuBackend::lg_basis_eq(F128 gamma, const std::vector<F128>& rho) {
  if ((uint64_t(1) << rho.size()) != Q_) throw std::runtime_error("Ligerito basis size mismatch");
  lg_pend_fold_.active = lg_pend_switch_ = false;
  lg_last_level_ = false;
  lg_tail_f_.clear();
  lg_tail_b_.clear();
  lane_ = LaneStage();
  lane_.active = true;
  lane_.w.assign(1, F256::one());
  add_lane_term(gamma, rho);
  lg_n_ = Q_;
}

F128 GpuBackend::lg_eval_eq(const std::vector<F128>& zp) {
  if (!lane_.active || lane_.bound || (uint64_t(1) << zp.size()) != Q_)
    throw std::runtime_error("OOD evaluation expects the committed base vector");
  lane_.dots = lane_dots(zp);
  lane_.dot_point = zp;
  const std::vector<F128> e = build_eq(std::vector<F128>(zp.begin() + S.log_dim, zp.end()));
  F128 y;
  for (size_t l = 0; l < e.size(); ++l) y += e[l] * lane_.dots[l];
  return y;
}

void GpuBackend::lg_add_eq(F128 beta, const std::vector<F128>& zp) {
  if (!lane_.active || lane_.bound) throw std::runtime_error("basis update expects the base stage");
  add_lane_term(beta, zp);
}

// u0 = sum_t c_t sum_j e_t[2j] h_t[2j], u2 = sum_t c_t sum_j (e_t[2j] + e_t[2j+1]) (h_t[2j] + h_t[2j+1]):
// the message over the row pairs of lanes 2j and 2j + 1, summed over the rows.
Msg256 GpuBackend::lane_message() const {
  Msg256 m;
  for (const LaneTerm& t : lane_.terms) {
    F256 u0, u2;
    for (size_t j = 0; j + 1 < t.e.size(); j += 2) {
      u0 += t.e[j] * t.h[j];
      u2 += (t.e[j] + t.e[j + 1]) * (t.h[j] + t.h[j + 1]);
    }
    m.u0 += u0 * t.coef;
    m.u2 += u2 * t.coef;
  }
  return m;
}

void GpuBackend::lane_fold(F256 r) {
  for (LaneTerm& t : lane_.terms)
    for (std::vector<F256>* v : {&t.e, &t.h}) {
      for (size_t j = 0; j < v->size() / 2; ++j) (*v)[j] = (*v)[2 * j] + r * ((*v)[2 * j + 1] + (*v)[2 * j]);
      v->resize(v->size() / 2);
    }
  const size_t n = lane_.w.size();
  lane_.w.resize(2 * n);
  for (size_t l = 0; l < n; ++l) {
    lane_.w[n + l] = lane_.w[l] * r;
    lane_.w[l] = lane_.w[l] + lane_.w[n + l];
  }
  lane_.bound++;
}

// All lanes folded and the code switched, in two launches; the message over the switched pairs.
Msg256 GpuBackend::lane_switch() {
  scr_off_ = 0;
  LaneTerms lt;
  lt.n = (uint32_t)lane_.terms.size();
  lt.lo_bits = std::min(S.log_dim, 10u);
  // lambda, then the terms' row points; both factors of every term's eq in one launch
  std::vector<F128> args;
  std::vector<std::pair<size_t, size_t>> of;
  for (const F256& w : lane_.w) {
    args.push_back(w.c0);
    args.push_back(w.c1);
  }
  for (uint32_t t = 0; t < lt.n; ++t) {
    const std::vector<F128>& p = lane_.terms[t].row_point;
    of.emplace_back(args.size(), args.size() + lt.lo_bits);
    of.emplace_back(args.size() + lt.lo_bits, args.size() + p.size());
    args.insert(args.end(), p.begin(), p.end());
    lt.coef[t] = dev(lane_.terms[t].e[0] * lane_.terms[t].coef);
  }
  std::vector<F128d*> eq;
  const F256d* dw = reinterpret_cast<const F256d*>(eq_tables(std::move(args), of, eq));
  for (uint32_t t = 0; t < lt.n; ++t) {
    lt.lo[t] = eq[2 * t];
    lt.hi[t] = eq[2 * t + 1];
  }
  FusedPublish fp = fused_publish();
  {
    Mark mk(this, ST_LIGERITO);
    launch_lg_lane_fold(q_, dw, S.lanes, rows(), lane_part_, st_);
    launch_lg_lane_switch(lane_part_, lane_fold_groups(S.lanes, rows(), (uint64_t)sm_count()), lt, rows(), lf_[0], lb_[0], part_, st_, fp);
  }
  lane_ = LaneStage();
  lg_cur_ = 0;
  lg_n_ = 2 * rows();
  return message256(fp);
}

Msg256 GpuBackend::message256(const FusedPublish& fp) {
  auto v = read_published(fp.seq, 4);
  Msg256 m;
  m.u0 = F256(v[0], v[1]);
  m.u2 = F256(v[2], v[3]);
  return m;
}

// The message over neighbours of the last level's tail, u0 = sum f0 b0, u2 = sum (f0 + f1) (b0 + b1).
Msg256 GpuBackend::lg_tail_message() const {
  Msg256 m;
  for (size_t i = 0; i + 1 < lg_tail_f_.size(); i += 2) {
    m.u0 += lg_tail_f_[i] * lg_tail_b_[i];
    m.u2 += (lg_tail_f_[i] + lg_tail_f_[i + 1]) * (lg_tail_b_[i] + lg_tail_b_[i + 1]);
  }
  return m;
}

Msg256 GpuBackend::lg_message(size_t d) {
  if (lane_.active) {
    if (lane_.folded && d == 1) return lane_switch();
    if (lane_.folded || lane_.bound == S.log_batch || d != rows())
      throw std::runtime_error("the lane stage's messages pair lanes, then the switched entries");
    return lane_message();
  }
  if (!lg_tail_f_.empty()) {
    if (d != 1 && d != lg_n_) throw std::runtime_error("the last level's messages pair neighbours");
    return lg_tail_message();
  }
  if (lg_pend_switch_ && (d == 1 || 2 * lg_n_ == d)) {
    // code switch and the message over its pairs (2i, 2i + 1) in one pass
    lg_pend_switch_ = false;
    const int nx = lg_cur_ ^ 1;
    FusedPublish fp = fused_publish();
    {
      Mark mk(this, ST_LIGERITO);
      launch_lg_switch_msg(lf_[lg_cur_], lb_[lg_cur_], lg_n_, lf_[nx], lb_[nx], part_, st_, fp);
    }
    lg_cur_ = nx;
    lg_n_ *= 2;
    return message256(fp);
  }
  if (lg_pend_switch_) lg_flush_fold();  // a code switch followed by a message with other pairs
  if (lg_pend_fold_.active) {
    // fold and message in one pass
    const uint64_t n_out = lg_n_ / 2;
    const size_t dm = (d == 1 || n_out == d) ? 1 : d;
    const int nx = lg_cur_ ^ 1;
    // the last level's folds finish on the host once one block holds what is left
    const bool tail = lg_last_level_ && n_out == LG_TAIL && lg_pend_fold_.d == 1 && dm == 1;
    F256d* fo = tail ? reinterpret_cast<F256d*>(d_tail_) : lf_[nx];
    F256d* bo = tail ? fo + LG_TAIL : lb_[nx];
    FusedPublish fp = fused_publish();
    {
      Mark mk(this, ST_LIGERITO);
      launch_lg_fold_msg256(lf_[lg_cur_], lb_[lg_cur_], n_out, dev(lg_pend_fold_.r), lg_pend_fold_.d, dm, fo, bo, part_,
                            st_, fp);
    }
    lg_pend_fold_.active = false;
    lg_cur_ = nx;
    lg_n_ = n_out;
    const Msg256 m = message256(fp);
    if (tail) {
      const TailPair t = read_tail(2 * LG_TAIL);  // f's halves, then b's
      for (size_t i = 0; i < LG_TAIL; ++i) {
        lg_tail_f_.push_back(F256(t.a[2 * i], t.a[2 * i + 1]));
        lg_tail_b_.push_back(F256(t.b[2 * i], t.b[2 * i + 1]));
      }
    }
    return m;
  }
  if (d == 1 || lg_n_ == d) d = 1;
  FusedPublish fp = fused_publish();
  { Mark mk(this, ST_LIGERITO); launch_lg_message256(lf_[lg_cur_], lb_[lg_cur_], lg_n_, d, part_, st_, fp); }
  return message256(fp);
}

void GpuBackend::lg_flush_fold() {
  if (lane_.active) throw std::runtime_error("the lane stage ends with its code switch and message");
  if (lg_pend_switch_) {
    lg_pend_switch_ = false;
    const int nx = lg_cur_ ^ 1;
    {
      Mark mk(this, ST_LIGERITO);
      launch_lg_code_switch(lf_[lg_cur_], lb_[lg_cur_], lg_n_, lf_[nx], lb_[nx], st_);
    }
    lg_cur_ = nx;
    lg_n_ *= 2;
  }
  if (!lg_pend_fold_.active) return;
  lg_pend_fold_.active = false;
  const uint64_t n_out = lg_n_ / 2;
  const int nx = lg_cur_ ^ 1;
  {
    Mark mk(this, ST_LIGERITO);
    launch_lg_fold256(lf_[lg_cur_], lb_[lg_cur_], n_out, dev(lg_pend_fold_.r), lg_pend_fold_.d, lf_[nx], lb_[nx],
                      st_);
  }
  lg_cur_ = nx;
  lg_n_ = n_out;
}

void GpuBackend::lg_fold(F256 r, size_t d) {
  if (lane_.active) {
    if (lane_.bound == S.log_batch || d != rows()) throw std::runtime_error("the lane stage folds lane pairs");
    lane_fold(r);
    return;
  }
  if (!lg_tail_f_.empty()) {
    if (d != 1) throw std::runtime_error("the last level folds neighbours");
    for (std::vector<F256>* v : {&lg_tail_f_, &lg_tail_b_}) {
      for (size_t i = 0; i < v->size() / 2; ++i) (*v)[i] = (*v)[2 * i] + r * ((*v)[2 * i + 1] + (*v)[2 * i]);
      v->resize(v->size() / 2);
    }
    lg_n_ /= 2;
    return;
  }
  lg_flush_fold();
  // held back: the next message runs fused with it, any other call performs it first
  lg_pend_fold_.active = true;
  lg_pend_fold_.r = r;
  lg_pend_fold_.d = d;
}

void GpuBackend::lg_code_switch() {
  if (lane_.active) {
    if (lane_.bound != S.log_batch) throw std::runtime_error("code switch before the last lane fold");
    lane_.folded = true;
    return;
  }
  lg_flush_fold();
  if (2 * lg_n_ > 2 * rows()) throw std::runtime_error("code switch exceeds the Ligerito buffers");
  lg_pend_switch_ = true;  // performed by the next message, or by lg_flush_fold
}

void GpuBackend::lg_commit(uint32_t level, uint32_t log_cols, uint32_t log_lanes, uint32_t log_rate,
                           uint32_t cap_depth, std::vector<Hash>& cap) {
  lg_flush_fold();
  if (lg_n_ != (uint64_t(1) << (log_cols + log_lanes))) throw std::runtime_error("Ligerito commit size mismatch");
  lg_last_level_ = level == S.lig.r;
  if (levels_.size() < level + 1) levels_.resize(level + 1);
  Level& L = levels_[level];
  uint64_t block_len = uint64_t(1) << (log_cols + log_rate);
  uint32_t lanes = 1u << log_lanes;
  if (L.block_len != block_len || L.lanes != lanes) {
    if (L.mat) {
      cudaFree(L.mat);
      cudaFree(L.tree);
      device_bytes_ -= L.block_len * L.lanes * sizeof(F128d) + 2 * L.block_len * 32;
    }
    CUDA_OK(cudaMalloc(&L.mat, block_len * lanes * sizeof(F128d)));
    CUDA_OK(cudaMalloc(&L.tree, 2 * block_len * 32));
    device_bytes_ += block_len * lanes * sizeof(F128d) + 2 * block_len * 32;
    L.block_len = block_len;
    L.lanes = lanes;
  }
  const F128d* tw = twiddles(log_cols + log_rate);
  { Mark mk(this, ST_LIGERITO); launch_lg_replicate(lf_[lg_cur_], lg_n_, block_len * lanes, L.mat, st_); }
  { Mark mk(this, ST_LG_NTT); launch_ntt(L.mat, lanes, log_cols + log_rate, log_rate, tw, st_); }
  const FusedPublish fp = fused_publish();
  {
    Mark mk(this, ST_LG_MERKLE);
    launch_merkle(L.mat, lanes, block_len, cap_depth, L.tree, st_, d_open(size_t(32) << cap_depth), fp);
  }
  cap = read_cap(cap_depth, fp);
}

Msg256 GpuBackend::lg_introduce_eq(const std::vector<F128>& zp, F128& answer) {
  lg_flush_fold();
  scr_off_ = 0;
  if ((uint64_t(1) << zp.size()) != lg_n_) throw std::runtime_error("OOD point size mismatch");
  if (zp.empty()) throw std::runtime_error("OOD point of no coordinates");
  const std::vector<F128> rest(zp.begin() + 1, zp.end());
  const uint64_t pairs = lg_n_ / 2;
  const FusedPublish fp = fused_publish();
  if (lg_intro_eq_direct(pairs)) {
    const F128d* dp = upload(rest);
    Mark mk(this, ST_LIGERITO);
    launch_lg_intro_eq(lf_[lg_cur_], dp, (uint32_t)rest.size(), pairs, pend_, part_, st_, fp);
  } else {
    EqSplit e = eq_split(rest, F128::one(), 10);
    Mark mk(this, ST_LIGERITO);
    launch_lg_intro_eq(lf_[lg_cur_], e.lo, e.lo_bits, e.hi, pairs, pend_, part_, st_, fp);
  }
  auto v = read_published(fp.seq, 2);
  pend_induced_ = false;
  pend_n_ = pairs;
  pend_z_ = zp[0];
  Msg256 m;
  const F128 even = (F128::one() + pend_z_) * v[0];
  answer = even + pend_z_ * v[1];
  m.u0 = F256(even);
  m.u2 = F256(v[0] + v[1]);
  return m;
}

Msg256 GpuBackend::lg_introduce_induced(uint32_t ln, uint32_t log_rate, const std::vector<uint64_t>& pos,
                                        const std::vector<F128>& w, const std::vector<std::vector<F128>>&) {
  lg_flush_fold();
  scr_off_ = 0;
  if ((uint64_t(2) << ln) != lg_n_) throw std::runtime_error("induced basis size mismatch");
  if (pos.size() != w.size()) throw std::runtime_error("induced basis: one weight per position");
  uint32_t log_d = ln + log_rate;
  for (uint64_t p : pos)
    if (p >> log_d) throw std::runtime_error("induced basis: position outside the codeword");
  uint32_t nq = (uint32_t)w.size();
  // queries that share a block of the sparse layers together (the weights' order does not matter)
  const uint32_t sparse = lg_sparse_layers(log_d, log_rate);
  std::vector<uint32_t> order(nq), start;
  for (uint32_t q = 0; q < nq; ++q) order[q] = q;
  if (sparse) std::sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return pos[a] < pos[b]; });
  std::vector<uint64_t> sp;
  std::vector<F128> sw;
  for (uint32_t q = 0; q < nq; ++q) {
    if (!q || (pos[order[q]] >> sparse) != (sp.back() >> sparse)) start.push_back(q);
    sp.push_back(pos[order[q]]);
    sw.push_back(w[order[q]]);
  }
  const uint32_t n_groups = (uint32_t)start.size();
  start.push_back(nq);
  const uint64_t* dpos = static_cast<const uint64_t*>(upload(sp.data(), sp.size() * 8));
  const F128d* dw = upload(sw);
  const uint32_t* dstart = static_cast<const uint32_t*>(upload(start.data(), start.size() * 4));
  F128d* y = static_cast<F128d*>(scratch(size_t(16) << log_d));
  const F128d* tw = twiddles(log_d);
  FusedPublish fp = fused_publish();
  {
    Mark mk(this, ST_LIGERITO);
    launch_lg_induced(dpos, dw, nq, dstart, n_groups, ln, log_rate, tw, lf_[lg_cur_], y, pend_, part_, st_, fp);
  }
  auto v = read_published(fp.seq, 2);
  pend_induced_ = true;
  pend_n_ = uint64_t(1) << ln;
  Msg256 m;
  m.u0 = F256(v[0]);
  m.u2 = F256(v[1], v[1]);
  return m;
}

void GpuBackend::lg_glue(F128 beta) {
  lg_flush_fold();
  Mark mk(this, ST_LIGERITO);
  const F128 odd = beta * pend_z_;
  launch_lg_glue(lb_[lg_cur_], pend_, dev(pend_induced_ ? beta : beta + odd), dev(odd), pend_n_, pend_induced_, st_);
}

void GpuBackend::lg_open(uint32_t level, const std::vector<uint64_t>& pos, uint32_t cap_depth,
                         std::vector<std::vector<F128>>& rows, std::vector<Hash>& paths) {
  lg_flush_fold();
  scr_off_ = 0;
  const F128d* mat;
  const uint8_t* tree;
  uint32_t lanes;
  uint64_t n_leaves;
  if (level == 0) { mat = cw0_; tree = tree0_; lanes = S.lanes; n_leaves = n_pos0_; }
  else { mat = levels_.at(level).mat; tree = levels_.at(level).tree; lanes = levels_[level].lanes; n_leaves = levels_[level].block_len; }
  uint32_t n = (uint32_t)pos.size();
  for (uint64_t p : pos)
    if (p >= n_leaves) throw std::runtime_error("opening position out of range");
  uint32_t depth = 0;
  while ((uint64_t(1) << depth) < n_leaves) ++depth;
  uint32_t plen = depth - cap_depth;
  const uint64_t* dpos = static_cast<const uint64_t*>(upload(pos.data(), n * 8));
  const size_t row_bytes = (size_t)n * lanes * 16, path_bytes = (size_t)n * plen * 32;
  uint8_t* d = d_open(row_bytes + path_bytes);
  const FusedPublish fp = fused_publish();
  {
    Mark mk(this, ST_LIGERITO);
    launch_gather_open(mat, lanes, tree, n_leaves, dpos, n, cap_depth, reinterpret_cast<F128d*>(d), d + row_bytes, st_, fp);
  }
  wait_published(fp.seq, true);
  d2h_ += row_bytes + path_bytes;
  const F128* hr = reinterpret_cast<const F128*>(h_open_);
  const Hash* hp = reinterpret_cast<const Hash*>(h_open_ + row_bytes);
  for (uint32_t q = 0; q < n; ++q) rows.emplace_back(hr + (size_t)q * lanes, hr + (size_t)(q + 1) * lanes);
  paths.insert(paths.end(), hp, hp + (size_t)n * plen);
}

std::vector<F256> GpuBackend::lg_residual() {
  if (!lg_tail_f_.empty()) return lg_tail_f_;
  lg_flush_fold();
  std::vector<F256> out(lg_n_);
  CUDA_OK(cudaMemcpyAsync(out.data(), lf_[lg_cur_], lg_n_ * sizeof(F256d), cudaMemcpyDeviceToHost, st_));
  d2h_ += lg_n_ * sizeof(F256d);
  sync();
  return out;
}

}  // namespace gpu
}  // namespace flock
