// Test harness: the device bytes that a backend counts and the estimate made without it, against what
// the device's free memory shows. A union's backend has the jagged assist's vectors beside its own.
// Test infrastructure only.
//
//   device_bytes <nu> <count of Keccak-f> <of SHA-256> <of BLAKE3>
#include "../../flock_gb300/csrc/gpu/backend.h"
#include <cstdio>

using namespace flock;

static ProveResult prove(const Statement& S, gpu::GpuBackend& G) {
  std::vector<std::vector<uint8_t>> in;
  std::vector<const uint8_t*> ptr;
  for (const SlotInfo& t : S.slots) {
    in.emplace_back(std::max<size_t>(1, t.count * input_record_bytes(t.hash)), uint8_t(0x5A));
    ptr.push_back(in.back().data());
  }
  G.begin_prove(nullptr);
  return prove_fast(S, G, ptr, reinterpret_cast<const uint8_t*>("bytes"), 5);
}
static uint64_t free_bytes() {
  size_t f = 0, total = 0;
  CUDA_OK(cudaDeviceSynchronize());
  CUDA_OK(cudaMemGetInfo(&f, &total));
  return f;
}

int main(int argc, char** argv) {
  if (argc != 5) return 2;
  try {
    const uint32_t nu = (uint32_t)atoi(argv[1]);
    std::vector<uint64_t> counts;
    for (int i = 2; i < 5; ++i) counts.push_back(strtoull(argv[i], nullptr, 0));
    const std::vector<HashKind> kinds = {HASH_KECCAK, HASH_SHA256, HASH_BLAKE3};  // slot order
    const Statement small = make_union_statement(kinds, 6, {3, 2, 1}), S = make_union_statement(kinds, nu, counts);
    {
      gpu::GpuBackend warm(small);  // the context, and every kernel of a union proof
      prove(small, warm);
    }
    const uint64_t before = free_bytes();
    gpu::GpuBackend G(S);
    prove(S, G);
    const uint64_t held = before - free_bytes(), counted = G.device_bytes();
    printf("held %llu counted %llu estimate %llu dense_words %llu\n", (unsigned long long)held, (unsigned long long)counted,
           (unsigned long long)gpu::GpuBackend::estimate_device_bytes(S), (unsigned long long)S.committed_words);
  } catch (const std::exception& e) {
    printf("FAILED: %s\n", e.what());
    return 1;
  }
  return 0;
}
