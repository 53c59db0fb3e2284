// frame_buffers.h -- who owns which page-locked buffer of an output frame
// (plain C++, so that it is checked on the host with other allocators).
#pragma once
#include <cstddef>
#include <cstdlib>
#include <list>
#include <mutex>
#include <unordered_map>

namespace agx {

// Each scenario that is bound for output has one buffer.  A caller may take it
// as it is (TAKEN bytes in all, beyond that callers copy); the scenario's next
// frame then needs another, and one given back is kept for that (288 MB: 2.9
// ms a frame, 12.7 with a buffer page-locked for each, 27 copied).  Kept are,
// of each size, as many as its scenarios are without and two a scenario beyond
// those (a caller that replaces its last frame by the next holds two), KEEP
// bytes of the latter in all, the oldest going first; of a size no scenario
// has any more, none.  A loop that takes and gives back within these bounds
// neither page-locks nor frees.
// Where no more memory can be page-locked the kept buffers are released; a
// scenario that still gets none has its frames in pageable memory (slower to
// copy to, never a caller's), so a run that could be bound does not fail later.
// Safe from several threads.
class FrameBuffers {
 public:
  static constexpr size_t KEEP = 1u << 30;
  static constexpr size_t TAKEN = 1u << 30;     // bytes callers may hold
  typedef float* (*Alloc)(size_t bytes);        // null: no memory
  typedef void (*Free)(float* p);
  FrameBuffers(Alloc alloc, Free release) : alloc_(alloc), free_(release) {}

  // a scenario is bound with frames of this size: its buffer, or null
  float* enter(size_t bytes) {
    {
      std::lock_guard<std::mutex> lock(mu_);
      sizes_[bytes].bound++;
    }
    float* p = get(bytes, true);
    if (!p) leave(nullptr, bytes);
    return p;
  }

  // it is bound no more; p: its buffer (null: taken)
  void leave(float* p, size_t bytes) {
    std::list<Kept> gone;
    {
      std::lock_guard<std::mutex> lock(mu_);
      Size& z = sizes_[bytes];
      z.bound--;
      if (p) {
        z.owned--;
        const auto it = live_.find(p);
        if (it->second.pageable) {
          live_.erase(it);
          std::free(p);
        } else {
          keep(p, bytes);
        }
      }
      trim(bytes, gone);
    }
    for (const Kept& k : gone) free_(k.p);
  }

  // a buffer for a scenario whose last one was taken; `lock`: page-locked or null
  float* get(size_t bytes, bool lock = false) {
    {
      std::lock_guard<std::mutex> guard(mu_);
      Size& z = sizes_[bytes];
      z.owned++;
      if (z.kept > 0) {
        auto it = kept_.end();                 // the latest: its pages are the likeliest in a cache
        while ((--it)->bytes != bytes) {
        }
        float* p = it->p;
        kept_.erase(it);
        z.kept--;
        return p;
      }
    }
    float* p = alloc_(bytes);
    if (!p) {
      release_kept();
      p = alloc_(bytes);
    }
    const bool pageable = !p && !lock;
    if (pageable) p = (float*)std::malloc(bytes);
    std::lock_guard<std::mutex> guard(mu_);
    if (p) live_[p] = {bytes, false, pageable};
    else sizes_[bytes].owned--;
    return p;
  }

  // a scenario's buffer becomes the caller's; false: the callers hold TAKEN
  // already, or it is not page-locked
  bool take(float* p) {
    std::lock_guard<std::mutex> lock(mu_);
    const auto it = live_.find(p);
    if (it == live_.end() || it->second.taken || it->second.pageable) return false;
    const size_t bytes = it->second.bytes;
    if (taken_bytes_ + bytes > TAKEN) return false;
    it->second.taken = true;
    taken_bytes_ += bytes;
    sizes_[bytes].owned--;
    return true;
  }

  // a caller's buffer comes back; any other pointer (one given back already,
  // one a scenario still owns) is left alone
  void give(float* p) {
    std::list<Kept> gone;
    {
      std::lock_guard<std::mutex> lock(mu_);
      const auto it = live_.find(p);
      if (it == live_.end() || !it->second.taken) return;
      it->second.taken = false;
      const size_t bytes = it->second.bytes;
      taken_bytes_ -= bytes;
      keep(p, bytes);
      trim(bytes, gone);
    }
    for (const Kept& k : gone) free_(k.p);
  }

 private:
  struct Size {
    long bound = 0;                      // scenarios with frames of this size
    long owned = 0;                      // those that have a buffer
    long kept = 0;
    long spare() const { return kept > bound - owned ? kept - (bound - owned) : 0; }
  };
  struct Live {
    size_t bytes;
    bool taken, pageable;
  };
  struct Kept {
    float* p;
    size_t bytes;
  };

  void keep(float* p, size_t bytes) {
    kept_.push_back({p, bytes});
    sizes_[bytes].kept++;
  }

  void drop(std::list<Kept>::iterator it, std::list<Kept>& gone) {
    live_.erase(it->p);
    sizes_[it->bytes].kept--;
    gone.splice(gone.end(), kept_, it);
  }

  void release_kept() {
    std::list<Kept> gone;
    {
      std::lock_guard<std::mutex> lock(mu_);
      while (!kept_.empty()) drop(kept_.begin(), gone);
    }
    for (const Kept& k : gone) free_(k.p);
  }

  // kept buffers beyond the bounds go: of this size, then the oldest of any
  void trim(size_t bytes, std::list<Kept>& gone) {
    Size& z = sizes_[bytes];
    size_t spare = 0;
    for (const auto& of : sizes_) spare += (size_t)of.second.spare() * of.first;
    for (auto it = kept_.begin(); it != kept_.end() && (z.spare() > 2 * z.bound || spare > KEEP);) {
      const auto at = it++;
      const Size& own = sizes_[at->bytes];
      if (own.spare() == 0 || (spare <= KEEP && at->bytes != bytes)) continue;
      spare -= at->bytes;
      drop(at, gone);
    }
    if (z.bound == 0) sizes_.erase(bytes);
  }

  std::mutex mu_;
  std::unordered_map<float*, Live> live_;          // every buffer
  std::unordered_map<size_t, Size> sizes_;         // those with scenarios
  std::list<Kept> kept_;                           // oldest first
  size_t taken_bytes_ = 0;
  const Alloc alloc_;
  const Free free_;
};

}  // namespace agx
