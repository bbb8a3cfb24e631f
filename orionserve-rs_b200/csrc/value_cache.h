// A bounded table of small values that are costly to make: the tensor maps of the launchers, by what they describe.
#pragma once

#include <cstddef>
#include <deque>
#include <map>
#include <mutex>

namespace orion {

// Values leave as copies, taken under the lock: a launch that needs several keeps what it has when a later lookup, its own or another
// thread's, has to make room. Room is made one value at a time, the oldest first, so that a full table costs a caller one value anew and not all.
template <typename Key, typename Value>
class ValueCache {
 public:
  explicit ValueCache(size_t most) : most_(most) {}
  // make(Value *) fills the value of a key that is not there. Its status is handed on, and nothing is kept unless that is 0.
  template <typename Make>
  int get(const Key &key, Value *out, Make make) {
    std::lock_guard<std::mutex> lock(mu_);
    auto it = values_.find(key);
    if (it == values_.end()) {
      Value v{};
      if (const int rc = make(&v)) return rc;
      if (values_.size() >= most_) {
        values_.erase(order_.front());
        order_.pop_front();
      }
      it = values_.emplace(key, v).first;
      order_.push_back(it);
    }
    *out = it->second;
    return 0;
  }

 private:
  const size_t most_;
  std::mutex mu_;
  std::map<Key, Value> values_;
  std::deque<typename std::map<Key, Value>::iterator> order_;  // as they came
};

}  // namespace orion
