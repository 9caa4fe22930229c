// Cache of resident block counts, safe with several threads.
#pragma once
#include <cstddef>
#include <map>
#include <mutex>
#include <tuple>

namespace ob {

// Keyed by all that the count depends on: the kernel (kernels of one signature share
// a function-pointer type, so by its address), the device, and the launch's block
// size and shared memory, which callers choose by grid.
class ResidentCache {
 public:
  template <class Count>
  int get(const void* kernel, int dev, int threads, std::size_t smem, Count&& count) {
    const Key key(kernel, dev, threads, smem);
    {
      std::lock_guard<std::mutex> lk(mu_);
      auto it = n_.find(key);
      if (it != n_.end()) return it->second;
    }
    const int n = count();
    std::lock_guard<std::mutex> lk(mu_);
    return n_.emplace(key, n).first->second;
  }

 private:
  using Key = std::tuple<const void*, int, int, std::size_t>;
  std::mutex mu_;
  std::map<Key, int> n_;
};

}  // namespace ob
