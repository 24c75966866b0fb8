// Launch configurations that depend on the device (SM count, kernel attributes,
// occupancy), found once per device of the process.  Host only.
#pragma once

#include <map>
#include <mutex>

namespace bilu {

template <class V>
class PerDevice {
 public:
  // *out = the value of `device`; make(&v), 0 on success, provides it on the first
  // call for that device (again if it failed).  Any thread.
  template <class F>
  int get(int device, V* out, F make) {
    std::lock_guard<std::mutex> lock(mu_);
    auto it = made_.find(device);
    if (it == made_.end()) {
      V v{};
      const int rc = make(&v);
      if (rc != 0) return rc;
      it = made_.emplace(device, v).first;
    }
    *out = it->second;
    return 0;
  }

 private:
  std::mutex mu_;
  std::map<int, V> made_;
};

}  // namespace bilu
