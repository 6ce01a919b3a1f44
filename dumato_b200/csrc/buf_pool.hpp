// Freed device buffers of one device, kept for the next owner. Host code only, with the driver's
// allocation calls passed in (its logic is tested without a GPU).
#pragma once

#include <cstddef>
#include <cstdint>
#include <functional>
#include <map>
#include <utility>

namespace dmb {

class BufPool {
 public:
  using Alloc = std::function<int(void**, size_t)>;  // 0 on success
  using Release = std::function<void(void*)>;

  BufPool(size_t max_bytes, Alloc alloc, Release release)
      : max_(max_bytes), alloc_(std::move(alloc)), release_(std::move(release)) {}

  // The smallest kept buffer of `bytes` to twice as many, else a new one. When the device has no room,
  // everything kept is released first.
  int take(void** p, size_t bytes) {
    auto it = kept_.lower_bound({bytes, 0});
    if (it != kept_.end() && it->first.first <= 2 * bytes) {
      *p = it->second;
      pooled_ -= it->first.first;
      age_.erase(it->first.second);
      kept_.erase(it);
      return 0;
    }
    int e = alloc_(p, bytes);
    if (e && drop()) e = alloc_(p, bytes);
    if (!e) size_[*p] = bytes;
    return e;
  }

  // Keeps the buffer, in place of the ones kept longest if they leave no room for it. False: not one of
  // this pool's.
  bool give(void* p) {
    auto it = size_.find(p);
    if (it == size_.end()) return false;
    const size_t bytes = it->second;
    if (bytes > max_) {
      size_.erase(it);
      release_(p);
      return true;
    }
    while (pooled_ + bytes > max_) evict(age_.begin()->second);
    const Key k{bytes, ++stamp_};
    kept_[k] = p;
    age_[k.second] = k;
    pooled_ += bytes;
    return true;
  }

  // Releases every kept buffer; the bytes released.
  size_t drop() {
    const size_t bytes = pooled_;
    while (!age_.empty()) evict(age_.begin()->second);
    return bytes;
  }

  size_t pooled() const { return pooled_; }

 private:
  using Key = std::pair<size_t, uint64_t>;  // size, time of return
  void evict(Key k) {
    auto it = kept_.find(k);
    size_.erase(it->second);
    release_(it->second);
    pooled_ -= k.first;
    age_.erase(k.second);
    kept_.erase(it);
  }

  size_t max_, pooled_ = 0;
  uint64_t stamp_ = 0;
  Alloc alloc_;
  Release release_;
  std::map<Key, void*> kept_;
  std::map<uint64_t, Key> age_;
  std::map<void*, size_t> size_;
};

}  // namespace dmb
