// A setting that the CUDA runtime keeps per device (a kernel's shared-memory
// limit), made once on each: a process may use several, and a limit set on one
// does not hold on another. Host code without CUDA.
#pragma once
#include <atomic>
#include <cstdint>

namespace gs {

class OncePerDevice {
  std::atomic<uint64_t> made_{0};  // bit d: made on device d

 public:
  // make() returns 0 when it succeeded; a failure is not remembered. Threads
  // that arrive together may each make it, which is harmless for a setting.
  template <class Make>
  int run(int device, Make&& make) {
    const bool kept = device >= 0 && device < 64;
    if (kept && (made_.load(std::memory_order_acquire) >> device & 1u)) return 0;
    const int error = make();
    if (error == 0 && kept) made_.fetch_or(uint64_t(1) << device, std::memory_order_release);
    return error;
  }
};

}  // namespace gs
