// Values made on demand and kept by key, for several threads; no CUDA in here, so that it is tested on the host.
#pragma once
#include <cstddef>
#include <mutex>
#include <unordered_map>

namespace b200 {

// At most `limit` entries: all are dropped when one more would be kept (callers that churn keys pay one rebuild each).
// A caller gets a copy of the value. A pointer into the map would dangle as soon as a later lookup, of the same launch or
// of another thread, dropped the entries.
template <class Key, class Value, class Hash>
class BoundedCache {
 public:
  explicit BoundedCache(size_t limit) : limit_(limit) {}

  // *out = the value of `key`. make(out) forms one that is missing; when it returns false nothing is kept.
  template <class Make>
  bool get(const Key& key, Value* out, Make make) {
    std::lock_guard<std::mutex> lock(mu_);
    auto it = map_.find(key);
    if (it != map_.end()) {
      *out = it->second;
      return true;
    }
    if (!make(out)) return false;
    if (map_.size() >= limit_) map_.clear();
    map_.emplace(key, *out);
    return true;
  }

  size_t size() {
    std::lock_guard<std::mutex> lock(mu_);
    return map_.size();
  }

 private:
  std::mutex mu_;
  std::unordered_map<Key, Value, Hash> map_;
  const size_t limit_;
};

}  // namespace b200
