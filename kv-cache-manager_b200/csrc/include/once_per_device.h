// Something that has to be done once on every device before it is relied on there, such as raising a kernel's limit of
// shared memory (a property of the kernel on one device).  Safe with several threads: two that come first both do it.
#pragma once
#include <atomic>

namespace kvcm {

class OncePerDevice {
 public:
  // `set` returns 0 when it has worked; what it returns else goes to the caller and is not kept.
  template <typename Set>
  int operator()(int device, Set set) {
    const bool known = device >= 0 && device < 64;                        // (beyond: every time)
    if (known && ((done_.load(std::memory_order_acquire) >> device) & 1)) return 0;
    const int rc = set();
    if (rc == 0 && known) done_.fetch_or(1ull << device, std::memory_order_release);
    return rc;
  }

 private:
  std::atomic<unsigned long long> done_{0};
};

}  // namespace kvcm
