// Host check of the output frames' buffer ownership (anuga_core_gb300/csrc/
// frame_buffers.h) with the C++ heap in place of page-locked memory: no buffer
// has two owners, whatever callers give back, and no steady loop page-locks.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <deque>
#include <functional>
#include <set>
#include <thread>
#include <vector>
#include "../../anuga_core_gb300/csrc/frame_buffers.h"

using agx::FrameBuffers;

constexpr size_t MB = 1u << 20;

static long g_bad = 0;
#define EXPECT(cond)                                              \
  do {                                                            \
    if (!(cond)) {                                                \
      std::printf("line %d: %s does not hold\n", __LINE__, #cond); \
      g_bad++;                                                    \
    }                                                             \
  } while (0)

static std::atomic<long> g_allocs{0}, g_frees{0};
static float* heap_alloc(size_t bytes) {
  g_allocs++;
  return (float*)std::malloc(bytes < 4096 ? bytes : 4096);      // no check writes further
}
static void heap_free(float* p) {
  g_frees++;
  std::free(p);
}
// the same where only `g_room` buffers can be page-locked
static long g_room = 0;
static std::set<float*> g_locked;
static float* scarce_alloc(size_t bytes) {
  if ((long)g_locked.size() >= g_room) return nullptr;
  float* p = heap_alloc(bytes);
  g_locked.insert(p);
  return p;
}
static void scarce_free(float* p) {
  EXPECT(g_locked.erase(p) == 1);
  heap_free(p);
}

// A buffer given back twice, one a scenario still owns, and a pointer that is
// no buffer: only a caller's buffer goes back.
static void check_give() {
  FrameBuffers B(heap_alloc, heap_free);
  const size_t n = 4000;
  float* a = B.enter(n);
  EXPECT(B.take(a));
  B.give(a);
  B.give(a);
  float* b = B.get(n);
  float* c = B.enter(n);
  EXPECT(b != c);
  B.give(b);                       // still the scenario's
  float* d = B.enter(n);
  EXPECT(d != b && d != c);
  float other = 0.0f;
  B.give(&other);
  B.give(nullptr);
  float* e = B.enter(n);
  EXPECT(e != &other && e != nullptr);
  float* own[] = {b, c, d, e};
  for (int i = 0; i < 4; i++)
    for (int j = 0; j < i; j++)
      if (own[i] == own[j]) return;       // (named above; freeing one twice would end the program)
  for (float* p : own) B.leave(p, n);
  EXPECT(g_allocs == g_frees);
}

// What a caller does with its frames: page-locks since the last call of this
// are counted by the checks below.  A scenario's frame as the library forms
// it (a buffer if the last was taken, then the copy to it), handed over or
// (null) copied.
struct Scenario {
  FrameBuffers& B;
  size_t bytes;
  float* own;
  Scenario(FrameBuffers& b, size_t n) : B(b), bytes(n), own(b.enter(n)) {}
  ~Scenario() { B.leave(own, bytes); }
  Scenario(const Scenario&) = delete;
  float* frame() {
    if (!own) own = B.get(bytes);
    float* p = own;
    if (!B.take(p)) return nullptr;
    own = nullptr;
    return p;
  }
};
static long allocs_of(const std::function<void()>& f) {
  const long before = g_allocs;
  f();
  return g_allocs - before;
}
static long live() { return g_allocs - g_frees; }

// Sizes no scenario has any more leave nothing behind, and so do not keep
// others from being kept.
static void check_dead_sizes() {
  FrameBuffers B(heap_alloc, heap_free);
  const long before = live();
  std::vector<float*> held;
  for (int i = 0; i < 8; i++) {
    Scenario s(B, (30u + i) * MB);
    held.push_back(s.frame());
  }
  for (float* p : held) B.give(p);
  EXPECT(live() == before);
  Scenario s(B, 72 * MB);
  EXPECT(allocs_of([&] { for (int i = 0; i < 100; i++) B.give(s.frame()); }) == 0);
}

// A scenario that leaves takes none of the buffers others of its size use.
static void check_leave() {
  FrameBuffers B(heap_alloc, heap_free);
  Scenario a(B, 72 * MB);
  B.give(a.frame());
  { Scenario b(B, 72 * MB); }
  EXPECT(allocs_of([&] { for (int i = 0; i < 10; i++) B.give(a.frame()); }) == 0);
  {
    Scenario b(B, 72 * MB);
    for (int i = 0; i < 4; i++) {
      B.give(a.frame());
      B.give(b.frame());
    }
  }
  EXPECT(allocs_of([&] { for (int i = 0; i < 10; i++) B.give(a.frame()); }) == 0);
}

// `count` scenarios with frames of `bytes`, pass after pass, by callers that
// drop each frame, replace it by the next, replace a whole pass by the next
// or keep all.  Nothing is page-locked in a steady loop, what is page-locked
// stays bounded, and it is freed with the last scenario and frame.
static void check_callers(int count, size_t bytes, bool handed_over) {
  for (int style = 0; style < 4; style++) {
    FrameBuffers B(heap_alloc, heap_free);
    const long before = live();
    std::vector<float*> held, last(count, nullptr);
    long early = 0, late = 0, handed = 0;
    {
      std::deque<Scenario> S;
      for (int i = 0; i < count; i++) S.emplace_back(B, bytes);
      for (int pass = 0; pass < 12; pass++) {
        (pass < 4 ? early : late) += allocs_of([&] {
          for (auto& s : S)
            if (!s.own) s.own = B.get(bytes);       // all frames are started, then waited for
          std::vector<float*> now;
          for (int i = 0; i < count; i++) {
            float* p = S[i].frame();
            if (pass >= 4 && p) handed++;
            if (style == 0) B.give(p);
            if (style == 1) {
              B.give(last[i]);
              last[i] = p;
            }
            if (style == 2) now.push_back(p);
            if (style == 3 && p) held.push_back(p);
          }
          if (style == 2) {
            for (float* p : last) B.give(p);
            last = now;
          }
        });
        EXPECT((size_t)(live() - before) * bytes <= count * bytes + FrameBuffers::KEEP + FrameBuffers::TAKEN);
      }
      EXPECT(held.size() * bytes <= FrameBuffers::TAKEN);
      if (style < 3) EXPECT(late == 0);
      if (style < 3) EXPECT(early <= 2 * count);
      if (style < 3 && handed_over) EXPECT(handed == 8 * count);
    }
    for (float* p : held) B.give(p);
    for (float* p : last) B.give(p);
    EXPECT(live() == before);
  }
}

// The oldest kept buffers make room, of whatever size: a scenario whose frames
// are no longer asked for does not keep another's from being kept.
static void check_room() {
  FrameBuffers B(heap_alloc, heap_free);
  const long before = live();
  {
    Scenario a(B, 300 * MB), b(B, 301 * MB), c(B, 302 * MB), d(B, 303 * MB);
    for (Scenario* s : {&a, &b, &c, &d})
      for (int i = 0; i < 3; i++) {
        float* p = s->frame();
        float* q = (s->own = B.get(s->bytes), s->frame());
        B.give(p);
        B.give(q);
        s->own = B.get(s->bytes);
      }
    EXPECT((live() - before - 4) * 300 * MB <= FrameBuffers::KEEP);
    EXPECT(allocs_of([&] {
             for (int i = 0; i < 10; i++) {
               B.give(d.frame());
               d.own = B.get(d.bytes);
             }
           }) == 0);
  }
  EXPECT(live() == before);
}

// No more memory can be page-locked: kept buffers make room, then frames go
// through pageable memory and are not handed over; a scenario that cannot be
// bound says so.
static void check_scarce() {
  FrameBuffers B(scarce_alloc, scarce_free);
  g_room = 3;
  {
    Scenario a(B, 4000);
    EXPECT(a.own != nullptr);
    float* p = a.frame();
    float* q = (a.own = B.get(a.bytes), a.frame());
    a.own = B.get(a.bytes);
    EXPECT(p && q && a.own && p != q && g_locked.size() == 3);
    B.give(q);                                    // kept: the next size may have its room
    {
      Scenario b(B, 8000);
      EXPECT(b.own != nullptr && g_locked.size() == 3);
      float* r = b.frame();
      EXPECT(r != nullptr);
      b.own = B.get(b.bytes);                     // all three are in use
      EXPECT(b.own != nullptr && g_locked.count(b.own) == 0);
      if (b.own) {
        b.own[0] = 1.0f;
        float* own = b.own;
        EXPECT(b.frame() == nullptr && b.own == own);
        B.give(own);                              // not a caller's
        EXPECT(b.own[0] == 1.0f);
      }
      EXPECT(B.enter(8000) == nullptr);           // binding needs a page-locked one, as ever
      B.give(r);
      EXPECT(g_locked.size() == 3);
    }
    EXPECT(g_locked.size() == 2);
    B.give(p);
  }
  EXPECT(g_locked.empty());
}

// Several threads, each with its own scenarios and frames: no buffer is in
// two hands (each writes its mark over what it holds and finds it again).
static void check_threads() {
  FrameBuffers B(heap_alloc, heap_free);
  std::atomic<long> mixed{0};
  std::vector<std::thread> T;
  for (int t = 0; t < 8; t++)
    T.emplace_back([&, t] {
      for (int round = 0; round < 200; round++) {
        Scenario s(B, 64 + 64 * (round % 3));
        std::vector<float*> held;
        for (int i = 0; i < 10; i++) {
          if (!s.own) s.own = B.get(s.bytes);
          s.own[0] = (float)(t * 100 + i);
          float* p = s.frame();
          if (p) held.push_back(p);
          if (p && p[0] != (float)(t * 100 + i)) mixed++;
          if (i % 3 == 2)
            while (!held.empty()) {
              B.give(held.back());
              held.pop_back();
            }
        }
        for (float* p : held) B.give(p);
      }
    });
  for (auto& t : T) t.join();
  EXPECT(mixed == 0);
}

int main() {
  check_give();
  check_dead_sizes();
  check_leave();
  check_callers(1, 72 * MB, true);
  check_callers(1, 288 * MB, true);      // 16M triangles
  check_callers(12, 31 * MB, true);      // 20.9M triangles in all
  check_callers(48, 31 * MB, false);     // beyond the bounds: part of them are copied
  check_callers(1, 1600 * MB, false);    // one frame beyond it: all are
  check_callers(3, 4000, true);
  check_room();
  check_scarce();
  check_threads();
  std::printf("failures %ld\n", g_bad);
  return g_bad ? 1 : 0;
}
