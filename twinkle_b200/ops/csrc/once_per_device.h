// Set-up that belongs to a device, such as a kernel's shared-memory limit: done at the first call on each device of the process, from any thread.
#pragma once
#include <atomic>
#include <cstdint>

namespace tk {

class OncePerDevice {
  std::atomic<uint64_t> done_{0};   // bit per device

 public:
  // Runs f unless it has already returned for this device.  Threads that arrive together may both run it; one that throws leaves the device to the next.
  template <typename F>
  void operator()(int device, F&& f) {
    const uint64_t bit = device >= 0 && device < 64 ? uint64_t{1} << device : 0;      // devices beyond are set up each time
    if (done_.load(std::memory_order_acquire) & bit) return;
    f();
    done_.fetch_or(bit, std::memory_order_release);
  }
};

}  // namespace tk
