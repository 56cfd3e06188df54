// Test harness: the zerocheck's folds on the CUDA backend beside the CPU oracle, for a point whose
// high coordinate is 0 or 1. A transcript draws such a coordinate with probability 2^-127, the
// weighted rounds cannot divide by its eq weight, and the backend takes the plain rounds, at any
// size. Test infrastructure only.
//
//   plain_rounds <hash 0|1|2> <n_blocks> <coordinate from the top> <0|1, or 2: left as drawn>
#include "../../flock_gb300/csrc/gpu/backend.h"
#include "../../oracle/cpu_backend.h"
#include <cstdio>

using namespace flock;

static uint64_t g_state = 0x9E3779B97F4A7C15ull;
static uint64_t next64() {
  uint64_t z = (g_state += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
static F128 draw() {
  const uint64_t lo = next64();
  return F128(lo, next64());
}
static void same(const char* what, uint32_t round, F128 a, F128 b) {
  if (a == b) return;
  printf("MISMATCH in %s, round %u\n", what, round);
  throw std::runtime_error(what);
}

int main(int argc, char** argv) {
  if (argc != 5) return 2;
  const HashKind hash = (HashKind)atoi(argv[1]);
  const uint32_t n = (uint32_t)atoi(argv[2]), from_top = (uint32_t)atoi(argv[3]), value = (uint32_t)atoi(argv[4]);
  try {
    const Statement S = make_statement(hash, n);
    std::vector<uint8_t> in(input_record_bytes(hash) * n);
    for (size_t i = 0; i + 8 <= in.size(); i += 8) {
      const uint64_t v = next64();
      memcpy(&in[i], &v, 8);
    }
    oracle::CpuBackend C(S);
    gpu::GpuBackend G(S);
    G.begin_prove(nullptr);
    C.witness({in.data()});
    G.witness({in.data()});
    const uint32_t L = S.m - 7;
    std::vector<F128> point(L), w(64);
    for (F128& v : point) v = draw();
    for (F128& v : w) v = draw();
    if (value < 2) point[L - 1 - from_top] = value ? F128::one() : F128();
    F128 c1, ci, g1, gi;
    C.zc_fold_skip(w, point, c1, ci);
    G.zc_fold_skip(w, point, g1, gi);
    same("skip fold g1", 0, c1, g1);
    same("skip fold ginf", 0, ci, gi);
    for (uint32_t i = 0; i < L; ++i) {
      const F128 rho = draw();
      const std::vector<F128> rest(point.begin() + 1 + i, point.end());
      C.zc_fold(rho, rest, c1, ci);
      G.zc_fold(rho, rest, g1, gi);
      same("fold g1", i, c1, g1);
      same("fold ginf", i, ci, gi);
    }
    const F128 rho = draw();
    C.zc_final(rho, c1, ci);
    G.zc_final(rho, g1, gi);
    same("final a", L, c1, g1);
    same("final b", L, ci, gi);
  } catch (const std::exception& e) {
    printf("FAILED: %s\n", e.what());
    return 1;
  }
  printf("PLAIN ROUNDS OK\n");
  return 0;
}
