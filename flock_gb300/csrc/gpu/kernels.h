// Launchers of the sm_103a kernels behind the prove_fast backend. Every launcher runs
// on the caller's stream; none allocates device memory (the one-time constant uploads
// excepted: upload_zc_consts and the witness constants live in module memory).
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <stdexcept>
#include <string>
#include "field.cuh"
#include "plan.h"

#define CUDA_OK(x)                                                                          \
  do {                                                                                      \
    cudaError_t e__ = (x);                                                                  \
    if (e__ != cudaSuccess)                                                                 \
      throw std::runtime_error(std::string("CUDA error ") + cudaGetErrorString(e__) + " at " + \
                               __FILE__ + ":" + std::to_string(__LINE__));                  \
  } while (0)

namespace flock {
namespace gpu {

// Kernel launches made by this library (all threads); read through flock_gb300_launch_count.
uint64_t launch_count();
void note_launch();
constexpr int MAX_DEVICES = 64;
// Raises `kernel`'s dynamic shared-memory limit to `bytes` on the current device, once per
// (kernel, device, size); thread-safe (provers on several threads launch the same kernels).
void set_dynamic_smem(const void* kernel, int bytes);
#define LAUNCH_OK()                    \
  do {                                 \
    CUDA_OK(cudaGetLastError());       \
    ::flock::gpu::note_launch();       \
  } while (0)

int sm_count();
constexpr uint64_t GB300_SMS = 152;  // for sizes computed without a device

// In-kernel publication of a round message: the last block to finish (a device-wide
// ticket counter) XOR-reduces every block's partials, writes the message to mapped host
// memory and then the sequence number, on which the host waits instead of on a copy and a stream
// synchronisation. counter must be zero before the launch; the last block resets it.
struct FusedPublish {
  F128d* out = nullptr;        // mapped host memory (null: no publication)
  uint32_t* flag = nullptr;    // mapped host memory
  uint32_t* counter = nullptr; // device memory
  uint32_t seq = 0;
};

// witness.cu — writes chunk columns [0, used_chunks) of z, a, b
void upload_witness_constants();  // once per process (synchronous symbol copies)
void launch_witness(int hash, const void* d_inputs, uint32_t n_inst, uint32_t nu, F128d* z, F128d* a, F128d* b,
                    uint32_t used_chunks, cudaStream_t s);

// commit.cu
void launch_fill_lane_major(const F128d* q, F128d* cw, uint32_t lanes, uint32_t log_dim, uint32_t log_pos,
                            cudaStream_t s);
void launch_ntt(F128d* data, uint32_t lanes, uint32_t log_d, uint32_t start_layer, const F128d* tw, cudaStream_t s);
// Leaves and the levels up to the cap level (2^cap_depth nodes); the levels above it are
// not computed.
// With `cap` (mapped memory, 32 2^cap_depth bytes) the cap is also written there and published.
void launch_merkle(const F128d* rows, uint32_t lanes, uint64_t n_leaves, uint32_t cap_depth, uint8_t* tree,
                   cudaStream_t s, uint8_t* cap = nullptr, FusedPublish pub = FusedPublish());
void launch_pow(const uint32_t digest_le[8], uint32_t bits, uint64_t start, uint64_t count, unsigned long long* d_min,
                uint32_t* d_counter, unsigned long long* out, uint32_t* flag, uint32_t seq, cudaStream_t s);
// An opening of n positions into mapped memory, published: the rows (lanes words each) at rows, the
// sibling paths (depth - cap_depth nodes each) at paths.
void launch_gather_open(const F128d* mat, uint32_t lanes, const uint8_t* tree, uint64_t n_leaves, const uint64_t* d_pos,
                        uint32_t n, uint32_t cap_depth, F128d* rows, uint8_t* paths, cudaStream_t s, FusedPublish pub);

// sumcheck.cu. Kernels returning a block count wrote per-block partials of the stated
// width into `part` and, with a FusedPublish, publish their sum.
// The lo and hi tables of an eq split (lo unscaled, hi times scale) in one launch.
void launch_eq_split(const F128d* d_point, uint32_t lo_bits, uint32_t hi_bits, F128d scale, F128d* lo, F128d* hi,
                     cudaStream_t s);
void launch_reduce_pair(const F128d* pa, uint32_t na, uint32_t wa, const F128d* pb, uint32_t nb, uint32_t wb,
                        cudaStream_t s, FusedPublish pub);

// unit[64 s + i]: extension of row bit s at Lambda point i; wconst, pconst: see ZcConsts.
void upload_zc_consts(const uint8_t* unit, const F128d* wconst, const F128d* pconst);
// Round-1 partials: *nrows rows of P_ab of width 64 into part_ab, as many of s_hat_v_c of width 128
// into part_svc, each array with room for part_room entries (checked before the launches).
// Words of z, a and b from live_words on are zero (the zero tail of a single slot's chunk
// columns) and are not read. g: 2^(m - 7) words of scratch.
void launch_zc_round1(const F128d* a, const F128d* b, const F128d* z, uint32_t m, uint64_t live_words,
                      const F128d* eq_lo, uint32_t lo_bits, const F128d* eq_hi, F128d* g, F128d* part_ab,
                      F128d* part_svc, uint64_t part_room, uint32_t* nrows, cudaStream_t s);
uint32_t launch_zc_fold_skip(const F128d* a, const F128d* b, const F128d* w64, uint64_t n_words, const F128d* eq_lo,
                             uint32_t lo_bits, const F128d* eq_hi, F128d* part, cudaStream_t s, FusedPublish pub);       // width 2
// First multilinear fold (at rho) of the skip-folded a, b, computed from the bits; writes
// n_pairs * 2 words of each folded vector and the next message. tabs: 4096-word scratch.
// Pairs from live_pairs on have zero inputs: their outputs are written as zeros and they
// add nothing to the message.
uint32_t launch_zc_fold2(const F128d* a, const F128d* b, const F128d* w64, F128d rho, F128d* tabs, uint64_t n_pairs,
                         uint64_t live_pairs, const F128d* eq_lo, uint32_t lo_bits, const F128d* eq_hi, F128d* aout,
                         F128d* bout, F128d* part, cudaStream_t s, FusedPublish pub);                                     // width 2
// The weighted form (see the kernels; its chunks: zc_weighted_lo_bits in plan.h): the skip fold's
// message and the first fold with its message. eq_lo: eq
// over the chunk's low coordinates (of words, then of pairs), h: eq over the high ones.
uint32_t launch_zc_fold_skip_weighted(const F128d* a, const F128d* b, const F128d* w64, uint64_t n_words,
                                      uint32_t lo_bits, const F128d* eq_lo, const F128d* h, F128d* part,
                                      cudaStream_t s, FusedPublish pub);                                                   // width 2
uint32_t launch_zc_fold2_weighted(const F128d* a, const F128d* b, const F128d* w64, F128d rho, uint64_t n_pairs,
                                  uint64_t live_pairs, uint32_t lo_bits, const F128d* eq_lo, const F128d* h,
                                  F128d* aout, F128d* bout, F128d* part, cudaStream_t s, FusedPublish pub);                // width 2
// out[c] = prod_j f[2j + bit j of c] over n factor pairs.
void launch_factor_table(const F128d* f, uint32_t n, F128d* out, cudaStream_t s);
// eq_lo == nullptr: eq = 1; eq_hi == nullptr: eq(j) = eq_lo[j mod 2^lo_bits]; else the split eq.
// unweight (or null): factors of the folded a entries. Pairs from live_pairs on have zero
// inputs (zeros written, nothing added to the message).
uint32_t launch_pair_fold(const F128d* ain, const F128d* bin, uint64_t n_pairs, uint64_t live_pairs, F128d r,
                          const F128d* eq_lo, uint32_t lo_bits, const F128d* eq_hi, const F128d* unweight, F128d* aout,
                          F128d* bout, F128d* part, cudaStream_t s, FusedPublish pub);  // width 2

void launch_lc_eq_inner(const F128d* w64, const F128d* er, uint32_t K, F128d* eqi, cudaStream_t s);
// A matrix by columns on the device (at most 2^16 rows).
struct CscDev {
  const uint32_t* col_ptr = nullptr;
  const uint16_t* rows = nullptr;
};
void launch_csc_fold(const CscDev& A, const CscDev& B, uint32_t K, const F128d* eqi, F128d* outa, F128d* outb,
                     cudaStream_t s);
// Keccak-f block R1CS: writes the nonzero entries of ca = eq^T A_0 and cb = eq^T B_0 (the
// caller zeroes both K-word vectors first). rc = the 24 round constants, rho[a + 5 b] = the
// rotation offset of lane (a, b) mod 64.
struct KeccakColumnConsts {
  uint64_t rc[24];
  uint8_t rho[25];
};
void launch_keccak_lincheck_columns(const F128d* eqi, F128d* ca, F128d* cb, const KeccakColumnConsts& kc,
                                    cudaStream_t s);
// Row fold of the used chunk columns into zv and a copy of it (K entries, zero past the used
// columns); part holds part_cap entries (at least 128 a column).
void launch_lc_zvec(const F128d* z, uint32_t nu, uint32_t used_chunks, const F128d* eq_lo, uint32_t lo_bits,
                    const F128d* eq_hi, F128d* part, uint64_t part_cap, uint32_t K, F128d* zv, F128d* captured,
                    cudaStream_t s);
uint32_t launch_lc_start(const F128d* ca, const F128d* cb, F128d alpha, F128d beta, uint32_t pin, uint32_t K,
                         F128d* comb, const F128d* zv, F128d* part, cudaStream_t s, FusedPublish pub);                   // width 2
uint32_t launch_lc_round(const F128d* comb, const F128d* zv, uint32_t len, F128d r, F128d* comb_out, F128d* zv_out,
                         F128d* part, cudaStream_t s, FusedPublish pub);
// Union lincheck: one slot's weighted comb (out = weight (alpha ca + cb), + beta at pin),
// and the first message of a comb built that way.
void launch_lc_slot_comb(const F128d* ca, const F128d* cb, F128d alpha, F128d weight, F128d beta, uint32_t pin,
                         uint32_t K, F128d* out, cudaStream_t s);
uint32_t launch_lc_top_message(const F128d* comb, const F128d* zv, uint32_t K, F128d* part, cudaStream_t s, FusedPublish pub);  // width 2
uint32_t launch_lc_matrix_evals(const F128d* ca, const F128d* cb, const F128d* er, const F128d* zp, uint32_t K,
                                F128d* part, cudaStream_t s, FusedPublish pub);                                          // width 2
void launch_lc_s_hat_v(const F128d* zv, const F128d* et, uint32_t n_tail, cudaStream_t s, FusedPublish pub);

// The committed stack of a union with non-identity compaction, as at most four slot
// segments (dense [base, base + rows * cols), column-major, first column col_off).
struct JaggedSegs {
  uint32_t n = 0;
  uint64_t base[4] = {0, 0, 0, 0}, rows[4] = {1, 1, 1, 1}, cols[4] = {0, 0, 0, 0}, col_off[4] = {0, 0, 0, 0};
};
// segs == nullptr: the aligned layout (row = d mod 2^nu, col = d >> nu).
uint32_t launch_mo_build_w(const F128d* q, const F128d* er0, const F128d* ec0, const F128d* er1, const F128d* ec1,
                           const F128d* tables, uint32_t nu, uint64_t area, uint64_t n, F128d* w, F128d* part,
                           cudaStream_t s, FusedPublish pub, const JaggedSegs* segs = nullptr);                          // width 2

// rounds.cu: the multipoint assist over a general jagged layout (union proofs). Dual values
// out[i * n_points + j] of claim i (row points z_row[i * n ..), run weights w[i * n_runs ..)) at
// points[j * m ..); runs: (t_c, t_next) pairs of 64-bit words.
void launch_as_dual(const F128d* z_row, uint32_t n, const F128d* points, uint32_t m, uint32_t n_claims,
                    uint32_t n_points, const void* runs, const F128d* w, uint32_t n_runs, F128d* out, cudaStream_t s);
// The sumcheck's vectors abar and g (n entries, abar zero from `area` on) and its first message.
void launch_as_build(const F128d* er0, const F128d* ec0, const F128d* er1, const F128d* ec1, const F128d* eq_lo,
                     uint32_t lo_bits, const F128d* eq_hi, const F128d* table, uint64_t area, uint64_t n,
                     const JaggedSegs& segs, F128d* abar, F128d* g, F128d* part, cudaStream_t s, FusedPublish pub);

// The lane stage (see the kernels): lane dots h[l] = sum_p q[l 2^log_d + p] eq(p) as `splits`
// partial rows of width `lanes` (returned), the fold of every lane by lambda into lane_fold_groups(lanes, D) partial rows of D entries,
// and the switched vectors with their message.
uint32_t launch_lg_lane_dots(const F128d* q, uint32_t lanes, uint32_t log_d, const F128d* eq_lo, uint32_t lo_bits,
                             const F128d* eq_hi, F128d* part, uint64_t part_room, cudaStream_t s);
uint32_t lane_fold_groups(uint32_t lanes, uint64_t D, uint64_t sms);
void launch_lg_lane_fold(const F128d* q, const F256d* lambda, uint32_t lanes, uint64_t D, F256d* part, cudaStream_t s);
// b = sum of n terms coef eq(point), each point's eq as lo (lo_bits) x hi tables.
struct LaneTerms {
  static constexpr uint32_t MAX = 4;
  uint32_t n = 0, lo_bits = 0;
  const F128d *lo[MAX] = {}, *hi[MAX] = {};
  F256d coef[MAX] = {};
};
uint32_t launch_lg_lane_switch(const F256d* fpart, uint32_t groups, const LaneTerms& terms, uint64_t D, F256d* fo,
                               F256d* bo, F128d* part, cudaStream_t s, FusedPublish pub);  // width 4
uint32_t launch_lg_message256(const F256d* f, const F256d* b, uint64_t n, uint64_t d, F128d* part, cudaStream_t s,
                              FusedPublish pub = FusedPublish());
uint32_t launch_lg_fold_msg256(const F256d* f, const F256d* b, uint64_t n_out, F256d r, uint64_t d_fold, uint64_t d_msg,
                               F256d* fo, F256d* bo, F128d* part, cudaStream_t s, FusedPublish pub);  // width 4
void launch_lg_fold256(const F256d* f, const F256d* b, uint64_t n_out, F256d r, uint64_t d,
                       F256d* fo, F256d* bo, cudaStream_t s);
void launch_lg_code_switch(const F256d* f, const F256d* b, uint64_t n, F256d* fo, F256d* bo, cudaStream_t s);
// The code switch and the round message over the switched vectors with pairs one apart,
// in one pass; published like launch_lg_message256 (four words).
uint32_t launch_lg_switch_msg(const F256d* f, const F256d* b, uint64_t n, F256d* fo, F256d* bo, F128d* part, cudaStream_t s,
                              FusedPublish pub);
void launch_lg_replicate(const F256d* f, uint64_t msg, uint64_t total, F128d* mat, cudaStream_t s);
// The pending eq basis as t over z[1 ..] (n_vars coordinates at `point`, or its two tables), the sums
// of f's even and odd entries with it published; the first form where lg_intro_eq_direct says so.
bool lg_intro_eq_direct(uint64_t pairs);
void launch_lg_intro_eq(const F256d* f, const F128d* point, uint32_t n_vars, uint64_t pairs, F128d* pend, F128d* part,
                        cudaStream_t s, FusedPublish pub);
void launch_lg_intro_eq(const F256d* f, const F128d* eq_lo, uint32_t lo_bits, const F128d* eq_hi, uint64_t pairs,
                        F128d* pend, F128d* part, cudaStream_t s, FusedPublish pub);  // width 2
// pos and w in order of pos >> lg_sparse_layers(...), start[g] the first query of group g (one
// value of that; start[n_groups] = n_q); without sparse layers start is not read.
uint32_t lg_sparse_layers(uint32_t log_d, uint32_t log_rate);
uint32_t launch_lg_induced(const uint64_t* pos, const F128d* w, uint32_t n_q, const uint32_t* start, uint32_t n_groups,
                           uint32_t ln, uint32_t log_rate, const F128d* tw, const F256d* f, F128d* y, F128d* basis,
                           F128d* part, cudaStream_t s, FusedPublish pub);  // width 2
void launch_lg_glue(F256d* b, const F128d* p, F128d w0, F128d w1, uint64_t n, bool induced, cudaStream_t s);

// rounds.cu
struct EqDesc {
  uint32_t p_off, n;   // coordinates point[p_off .. p_off + n)
  uint64_t out_off;    // first entry in the output
};
// d_desc: the n_desc descriptors on the device, desc: the same on the host.
void launch_eq_tables(const F128d* point, const EqDesc* d_desc, const EqDesc* desc, uint32_t n_desc, F128d* out,
                      cudaStream_t s);

}  // namespace gpu
}  // namespace flock
