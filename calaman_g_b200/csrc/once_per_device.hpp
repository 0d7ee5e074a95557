// once_per_device.hpp -- a step that is due once on every device of a process:
// a kernel's attributes belong to the device's context, so a second device needs
// them set again.
#pragma once

#include <atomic>

namespace clm {

class OncePerDevice {
  std::atomic<unsigned long long> done_{0};  // a bit per device

 public:
  // configure() (a status, 0: success) unless it has succeeded for `device`
  // before. Threads that race may both run it; devices past the 64th run it every
  // time.
  template <typename F>
  auto run(int device, F &&configure) -> decltype(configure()) {
    using Status = decltype(configure());
    const unsigned long long bit = device >= 0 && device < 64 ? 1ull << device : 0ull;
    if (done_.load(std::memory_order_acquire) & bit) return Status(0);
    const Status st = configure();
    if (st == Status(0)) done_.fetch_or(bit, std::memory_order_release);
    return st;
  }
};

}  // namespace clm
