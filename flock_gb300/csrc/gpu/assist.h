// The jagged multipoint assist's bulk steps on the device (union statements): own stream,
// buffers, staging and publication, since the assist's thread runs beside the inner open.
#pragma once
#include "kernels.h"
#include "../host/prover.h"

namespace flock {
namespace gpu {

class JaggedAssist : public JaggedAssistOps {
 public:
  JaggedAssist(const Statement& s, int device);
  ~JaggedAssist() override;
  JaggedAssist(const JaggedAssist&) = delete;
  JaggedAssist& operator=(const JaggedAssist&) = delete;
  void dual_values(const std::vector<AssistStatement>& unit, const std::vector<std::vector<F128>>& points, uint32_t m,
                   std::vector<std::vector<F128>>& values) override;
  void build(const std::vector<RsClaimPoint>& claims, const std::vector<F128>& scale, const std::vector<F128>& rho,
             const std::vector<F128>& table, F128& g1, F128& gi) override;
  void fold(F128 r, F128& g1, F128& gi) override;
  // Device bytes held, and the same without a device.
  uint64_t device_bytes() const { return device_bytes_; }
  static uint64_t estimate_device_bytes(const Statement& s, uint64_t sms);

 private:
  template <class T> T* alloc(size_t n);
  const void* upload(const void* src, size_t bytes);
  FusedPublish publish();
  void read(const FusedPublish& p, bool stage, F128& g1, F128& gi);

  const Statement& S;
  int device_;
  cudaStream_t st_ = nullptr;
  std::vector<void*> owned_;
  uint64_t device_bytes_ = 0;
  uint64_t n_ = 0;                               // dense words 2^m
  F128d *a_[3] = {}, *g_[3] = {};                // n, n/2 and n/4 entries: fold 0 -> 1 -> 2 -> 1 ...
  int cur_ = 0;
  uint64_t len_ = 0;                             // current length
  F128d *er_[2] = {}, *ec_[2] = {}, *eq_lo_ = nullptr, *eq_hi_ = nullptr, *part_ = nullptr, *out_ = nullptr;
  uint8_t *d_stage_ = nullptr, *h_stage_ = nullptr;
  size_t stage_cap_ = 0, stage_off_ = 0;
  F128d *h_pub_ = nullptr, *d_pub_ = nullptr, *h_out_ = nullptr;
  uint32_t *h_flag_ = nullptr, *d_flag_ = nullptr, *counter_ = nullptr, seq_ = 0;
};

// A statement that is not one full-height slot takes the assist.
inline bool takes_jagged_assist(const Statement& s) { return s.slots.size() != 1 || !s.identity; }
// The committed stack of a union as slot segments (at most four non-empty slots).
JaggedSegs jagged_segs(const Statement& S);

}  // namespace gpu
}  // namespace flock
