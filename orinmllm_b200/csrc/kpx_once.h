// A value that is worked out once per device and then read without a lock.
#pragma once
#include <stdint.h>

#include <atomic>
#include <mutex>

namespace kpx {

template <typename V>
class PerDevice {
 public:
  // The value of device `dev`.  The first caller works it out with make(V&); others wait for it.  It is
  // published whole and never written again.  nullptr if make returns false (asked again next time)
  // or the device is beyond the table.
  template <typename Make>
  const V* get(int dev, Make make) {
    if (dev < 0 || dev >= 64) return nullptr;
    const uint64_t bit = uint64_t(1) << dev;
    if (!(done_.load(std::memory_order_acquire) & bit)) {
      std::lock_guard<std::mutex> lock(mu_);
      if (!(done_.load(std::memory_order_relaxed) & bit)) {  // (another thread may have been here meanwhile)
        V v{};
        if (!make(v)) return nullptr;
        values_[dev] = v;
        done_.fetch_or(bit, std::memory_order_release);
      }
    }
    return &values_[dev];
  }

 private:
  V values_[64]{};
  std::atomic<uint64_t> done_{0};
  std::mutex mu_;
};

}  // namespace kpx
