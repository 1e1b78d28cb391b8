// Attributes of kernels (shared memory above 48 KB, cluster sizes) belong to a
// function on one device: a process with handles on two GPUs sets them on both.
// This remembers what is set, per function, attribute and device, so that a launch
// on the hot path asks the runtime only once; safe with several threads.
#pragma once
#include <map>
#include <mutex>
#include <tuple>

namespace pmg {

class FuncAttrs {
  std::mutex mu;
  std::map<std::tuple<const void *, int, int>, int> set;

 public:
  // apply() returns 0 on success; a failed one is tried again by the next call
  template <typename Apply>
  int once(const void *fn, int attr, int device, int value, Apply apply) {
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_tuple(fn, attr, device);
    const auto it = set.find(key);
    if (it != set.end() && it->second == value) return 0;
    const int rc = (int)apply();
    if (rc == 0) set[key] = value;
    return rc;
  }
};

}  // namespace pmg
