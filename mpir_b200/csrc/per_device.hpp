// Work that is done once on each device (a kernel's attributes).
#pragma once
#include <atomic>
#include <cstdint>

namespace mpir {

class OncePerDevice {
 public:
  // f(), unless a call for this device has come back from it.  Threads that
  // are the first together each call it.
  template <class F>
  void run(int device, F f) {
    const uint64_t bit = device >= 0 && device < 64 ? uint64_t{1} << device : 0;
    if (done_.load(std::memory_order_acquire) & bit) return;
    f();
    done_.fetch_or(bit, std::memory_order_release);
  }

 private:
  std::atomic<uint64_t> done_{0};
};

}  // namespace mpir
