// per_device.h -- set-up of kernels, once per device (a header of its own that a
// host compiler takes too).
#pragma once

#include <stddef.h>

#include <map>
#include <mutex>
#include <tuple>

namespace pcc {

// A kernel's shared-memory limit and its resident CTAs per SM belong to the
// device that was current when they were set or queried; the calls take a
// driver lock that serialises concurrent contexts, so each is made once.
class PerDevice {
 public:
  // *value = what make(value) stored the first time for (device, key, size).
  // A make that answers false is not kept.
  template <class F>
  bool Get(int device, const void* key, size_t size, int* value, F make) {
    std::lock_guard<std::mutex> lk(mu_);
    const auto k = std::make_tuple(device, key, size);
    const auto it = values_.find(k);
    if (it != values_.end()) {
      *value = it->second;
      return true;
    }
    *value = 0;
    if (!make(value)) return false;
    values_.emplace(k, *value);
    return true;
  }

 private:
  std::mutex mu_;
  std::map<std::tuple<int, const void*, size_t>, int> values_;
};

}  // namespace pcc
