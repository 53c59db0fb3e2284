// frame_buffers.h -- who owns which page-locked buffer of an output frame
// (plain C++, so that it is checked on the host with other allocators).
#pragma once
#include <cstddef>
#include <mutex>
#include <unordered_map>
#include <unordered_set>
#include <vector>

namespace agx {

// A buffer belongs to a scenario or, once taken, to a caller; one given back
// is kept for the next frame of its size (page-locking 72 MB takes some 20
// ms), at most KEEP bytes in all, and those of a size are released with a
// scenario of that size.  Safe from several threads.
class FrameBuffers {
 public:
  static constexpr size_t KEEP = 256u << 20;
  static constexpr size_t TAKEN = 1u << 30;     // bytes callers may hold
  typedef float* (*Alloc)(size_t bytes);        // null: no memory
  typedef void (*Free)(float* p);
  FrameBuffers(Alloc alloc, Free release) : alloc_(alloc), free_(release) {}

  // a buffer for a scenario, or null
  float* get(size_t bytes) {
    {
      std::lock_guard<std::mutex> lock(mu_);
      auto it = kept_.find(bytes);
      if (it != kept_.end()) {
        float* p = it->second;
        kept_.erase(it);
        kept_bytes_ -= bytes;
        return p;
      }
    }
    float* p = alloc_(bytes);
    if (!p) return nullptr;
    std::lock_guard<std::mutex> lock(mu_);
    size_[p] = bytes;
    return p;
  }

  // a scenario's buffer becomes the caller's; false: the callers hold TAKEN already
  bool take(float* p) {
    std::lock_guard<std::mutex> lock(mu_);
    const size_t bytes = size_[p];
    if (taken_bytes_ + bytes > TAKEN) return false;
    taken_.insert(p);
    taken_bytes_ += bytes;
    return true;
  }

  // a caller's buffer comes back; any other pointer (one given back already,
  // one a scenario still owns) is left alone
  void give(float* p) {
    {
      std::lock_guard<std::mutex> lock(mu_);
      if (!taken_.erase(p)) return;
      auto it = size_.find(p);
      const size_t bytes = it->second;
      taken_bytes_ -= bytes;
      if (kept_bytes_ + bytes <= KEEP) {
        kept_.emplace(bytes, p);
        kept_bytes_ += bytes;
        return;
      }
      size_.erase(it);
    }
    free_(p);
  }

  // a scenario's buffer (may be null) and the kept ones of its size are freed
  void release(float* p, size_t bytes) {
    std::vector<float*> gone;
    {
      std::lock_guard<std::mutex> lock(mu_);
      if (p && size_.erase(p)) gone.push_back(p);
      for (auto it = kept_.find(bytes); it != kept_.end(); it = kept_.find(bytes)) {
        gone.push_back(it->second);
        size_.erase(it->second);
        kept_.erase(it);
        kept_bytes_ -= bytes;
      }
    }
    for (float* q : gone) free_(q);
  }

 private:
  std::mutex mu_;
  std::unordered_map<float*, size_t> size_;              // every live buffer
  std::unordered_multimap<size_t, float*> kept_;
  std::unordered_set<float*> taken_;
  size_t kept_bytes_ = 0, taken_bytes_ = 0;
  const Alloc alloc_;
  const Free free_;
};

}  // namespace agx
