// Launch configurations that depend on the device (SM count, kernel attributes,
// occupancy), found once per device of the process.  Host only.
#pragma once

#include <atomic>
#include <map>
#include <mutex>

namespace bilu {

template <class V>
class PerDevice {
 public:
  // *out = the value of `device`; make(&v), 0 on success, provides it on the first
  // call for that device (again if it failed).  Any thread; later calls for the
  // first kFast devices take no lock (a launch is a few microseconds).
  template <class F>
  int get(int device, V* out, F make) {
    const bool fast = device >= 0 && device < kFast;
    if (fast) {
      if (const V* v = ready_[device].load(std::memory_order_acquire)) {
        *out = *v;
        return 0;
      }
    }
    std::lock_guard<std::mutex> lock(mu_);
    auto it = made_.find(device);
    if (it == made_.end()) {
      V v{};
      const int rc = make(&v);
      if (rc != 0) return rc;
      it = made_.emplace(device, v).first;  // the map's nodes stay where they are
      if (fast) ready_[device].store(&it->second, std::memory_order_release);
    }
    *out = it->second;
    return 0;
  }

 private:
  static constexpr int kFast = 16;
  std::atomic<const V*> ready_[kFast] = {};
  std::mutex mu_;
  std::map<int, V> made_;
};

}  // namespace bilu
