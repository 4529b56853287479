// Settings that the CUDA runtime keeps per device, made once on each of them
// (compiles with or without CUDA).
#pragma once

#include <atomic>
#include <cstdint>

namespace pwmgpu {

// One for each setting, of static storage.  From any thread: run(device, set)
// returns 0 once set() has succeeded on that device; a set() that fails is
// tried again by the next call, and two threads may both make the setting.
class OncePerDevice {
 public:
  template <typename F>
  int run(int device, F&& set) {
    const uint64_t bit = device >= 0 && device < 64 ? uint64_t(1) << device : 0;  // others: every time
    if (done_.load(std::memory_order_acquire) & bit) return 0;
    const int error = set();
    if (error == 0) done_.fetch_or(bit, std::memory_order_release);
    return error;
  }

 private:
  std::atomic<uint64_t> done_{0};
};

}  // namespace pwmgpu
