// What a launch asks of the runtime once per configuration, kept by it (host
// code).  A configuration is a kernel, its block and shared memory and the
// device; there are as many as kernels and box depths, so every one is kept: a
// table that was full made each further configuration ask on every launch.
#pragma once

#include <cstddef>
#include <map>
#include <mutex>
#include <new>
#include <tuple>

namespace orsp {

class LaunchCache {
 public:
  // The value of a configuration, from ask(int *value), a status, at first.
  template <class Ask>
  int get(const void *fn, int threads, size_t smem, int device, int *value, Ask ask) {
    std::lock_guard<std::mutex> lock(mu_);
    const Key key(fn, threads, smem, device);
    const auto it = kept_.find(key);
    if (it != kept_.end()) {
      *value = it->second;
      return 0;
    }
    const int rc = ask(value);
    if (rc) return rc;
    try {
      kept_.emplace(key, *value);
    } catch (const std::bad_alloc &) {  // asked again next time
    }
    return 0;
  }

 private:
  using Key = std::tuple<const void *, int, size_t, int>;
  std::map<Key, int> kept_;
  std::mutex mu_;
};

}  // namespace orsp
