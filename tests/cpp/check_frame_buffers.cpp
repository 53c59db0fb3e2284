// Host check of the output frames' buffer ownership (anuga_core_gb300/csrc/
// frame_buffers.h) with the C++ heap in place of page-locked memory: no buffer
// has two owners, whatever callers give back.
#include <cstdio>
#include <cstdlib>
#include "../../anuga_core_gb300/csrc/frame_buffers.h"

using agx::FrameBuffers;

static long g_allocs = 0, g_frees = 0;
static float* heap_alloc(size_t bytes) {
  g_allocs++;
  return (float*)std::malloc(bytes);
}
static void heap_free(float* p) {
  g_frees++;
  std::free(p);
}

static long g_bad = 0;
#define EXPECT(cond)                                              \
  do {                                                            \
    if (!(cond)) {                                                \
      std::printf("line %d: %s does not hold\n", __LINE__, #cond); \
      g_bad++;                                                    \
    }                                                             \
  } while (0)

// A buffer given back twice, one a scenario still owns, and a pointer that is
// no buffer: only a caller's buffer goes back.
static void check_give() {
  FrameBuffers B(heap_alloc, heap_free);
  const size_t n = 4000;
  float* a = B.get(n);
  EXPECT(B.take(a));
  B.give(a);
  B.give(a);
  float* b = B.get(n);
  float* c = B.get(n);
  EXPECT(b != c);
  B.give(b);                       // still the scenario's
  float* d = B.get(n);
  EXPECT(d != b && d != c);
  float other = 0.0f;
  B.give(&other);
  B.give(nullptr);
  float* e = B.get(n);
  EXPECT(e != &other && e != nullptr);
  float* own[] = {b, c, d, e};
  for (int i = 0; i < 4; i++)
    for (int j = 0; j < i; j++)
      if (own[i] == own[j]) return;       // (named above; freeing it twice would end the program)
  for (float* p : own) B.release(p, n);
  EXPECT(g_allocs == g_frees);
}

int main() {
  check_give();
  std::printf("failures %ld\n", g_bad);
  return g_bad ? 1 : 0;
}
