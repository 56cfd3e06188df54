// Waiting for a sequence number that a kernel publishes into mapped host memory. No CUDA in here:
// the stream is a function, so that a host test can stand in for it.
#pragma once
#include <atomic>
#include <chrono>
#include <cstdint>
#include <stdexcept>
#include <string>
#include <thread>

namespace flock {
namespace gpu {

constexpr double ROUND_WAIT_MS = 20000;

// Spin until *flag is seq: a short hot spin for the common case of a message a few microseconds
// away, then a spin that yields the core on every pass, so that concurrent provers' host work
// (assists, transcripts) is not starved by waiting threads. running() says whether the stream
// still has work (and throws its error). A round's message is reported as stalled after limit_ms;
// the result of a whole stage (stage: a cap, an opening, round 1, the assist's build) is waited
// for as long as the stream runs, as a stream synchronisation would, and then for limit_ms.
template <class Running>
void wait_published_flag(const volatile uint32_t* flag, uint32_t seq, bool stage, double limit_ms, Running running) {
  using Clock = std::chrono::steady_clock;
  uint64_t spins = 0;
  Clock::time_point t0;
  bool timed = false;
  while (*flag != seq) {
    ++spins;
    if (spins > 2048) std::this_thread::yield();
    if ((spins & 0x3FFF) == 0) {
      const bool busy = running();
      const Clock::time_point t = Clock::now();
      if (!timed || (stage && busy)) {
        t0 = t;
        timed = true;
      } else if (std::chrono::duration<double, std::milli>(t - t0).count() > limit_ms) {
        throw std::runtime_error("device result not published within " + std::to_string((int)(limit_ms / 1000)) + " s");
      }
    }
  }
  std::atomic_thread_fence(std::memory_order_acquire);
}

}  // namespace gpu
}  // namespace flock
