// The wait for a published sequence number (csrc/gpu/wait.h), with a function in the stream's place
// and a limit of 50 ms: a flag that nobody sets is an error at the limit in a round, and in a
// stage only once the stream has nothing left to run.
#include "../../flock_gb300/csrc/gpu/wait.h"
#include <cstdio>

using namespace flock::gpu;
using Clock = std::chrono::steady_clock;

static int failures = 0;
static void expect(bool ok, const char* what) {
  if (!ok) { ++failures; printf("%s\n", what); }
}
static double ms_since(Clock::time_point t) { return std::chrono::duration<double, std::milli>(Clock::now() - t).count(); }

constexpr double LIMIT = 50;
// Milliseconds until the wait gave up (or came back: done = true).
template <class Running>
static double wait_for(volatile uint32_t* flag, bool stage, bool& done, Running running) {
  const auto t = Clock::now();
  done = true;
  try {
    wait_published_flag(flag, 7, stage, LIMIT, running);
  } catch (const std::runtime_error&) {
    done = false;
  }
  return ms_since(t);
}

int main() {
  bool done;
  {
    volatile uint32_t flag = 7;
    wait_for(&flag, false, done, [] { return true; });
    expect(done, "a flag that is set already");
  }
  {
    volatile uint32_t flag = 6;
    const double ms = wait_for(&flag, false, done, [] { return true; });
    expect(!done && ms >= LIMIT, "a round on a running stream ends at the limit");
  }
  {
    volatile uint32_t flag = 6;
    const double ms = wait_for(&flag, true, done, [] { return false; });
    expect(!done && ms >= LIMIT, "a stage on an idle stream ends at the limit");
  }
  {
    volatile uint32_t flag = 6;
    const auto t = Clock::now();
    const double ms = wait_for(&flag, true, done, [&] {
      if (ms_since(t) < 6 * LIMIT) return true;
      flag = 7;  // the kernel publishes at its end
      return false;
    });
    expect(done && ms >= 6 * LIMIT, "a stage is waited for while the stream runs");
  }
  {
    volatile uint32_t flag = 6;
    const auto t = Clock::now();
    auto last_busy = t;  // the limit counts from the last time the stream was seen to run
    wait_for(&flag, true, done, [&] {
      if (ms_since(t) >= 3 * LIMIT) return false;
      last_busy = Clock::now();
      return true;
    });
    expect(!done && ms_since(t) >= 3 * LIMIT && ms_since(last_busy) >= LIMIT, "a stage that ends without its flag is an error");
  }
  {
    volatile uint32_t flag = 6;
    bool thrown = false;
    try {
      wait_published_flag(&flag, 7, true, LIMIT, []() -> bool { throw std::logic_error("stream"); });
    } catch (const std::logic_error&) {
      thrown = true;
    }
    expect(thrown, "the stream's error comes through");
  }
  printf("failures %d\n", failures);
  return failures != 0;
}
