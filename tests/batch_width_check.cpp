// Host check of the batched kernel's width rule (csrc/batch_width.hpp) on a GPU of 148 SMs: the width
// that was measured faster where the sides differ, and the numbers of the call it goes by.
#include <cstdio>

#include "batch_width.hpp"

static int failures = 0;
#define EXPECT(c) \
  do { \
    if (!(c)) { \
      ++failures; \
      std::printf("line %d: %s\n", __LINE__, #c); \
    } \
  } while (0)

using sov::BatchCall;

static BatchCall uniform(int count, int m, int n) {
  BatchCall c;
  for (int i = 0; i < count; ++i) c.add(m, n);
  return c;
}
static int width(const BatchCall& c, int m) { return sov::width_for(148, c, sov::bucket_of(m)); }
// transportation LPs with lo .. hi sources and sinks
static BatchCall mixed(int count, int lo, int hi) {
  BatchCall c;
  unsigned s = 12345;
  auto next = [&] { return lo + static_cast<int>((s = s * 1664525u + 1013904223u) >> 8) % (hi - lo + 1); };
  for (int i = 0; i < count; ++i) {
    const int a = next(), b = next();
    c.add(a + b, a * b);
  }
  return c;
}

int main() {
  EXPECT(width(uniform(1, 100, 2500), 100) == 512 && width(uniform(148, 36, 324), 36) == 512);
  EXPECT(width(uniform(149, 36, 324), 36) == 256 && width(uniform(296, 70, 1225), 70) == 256);
  // one size, up to four LPs an SM: all on the GPU at once
  for (int count : {297, 350, 444, 520, 592})
    for (int n : {64, 256, 324, 576, 900}) EXPECT(width(uniform(count, 60, n), 60) == 128);
  EXPECT(width(uniform(350, 80, 1600), 80) == 128 && width(uniform(444, 120, 1100), 120) == 128);
  EXPECT(width(uniform(592, 120, 1100), 120) == 256 && width(uniform(592, 100, 2500), 100) == 256);
  // beyond: by rows and columns
  for (int count : {593, 1000, 1500, 3000, 4096, 4700})
    for (int n : {91, 324, 576, 900}) EXPECT(width(uniform(count, 60, n), 60) == 128);
  EXPECT(width(uniform(1000, 120, 300), 120) == 128 && width(uniform(1500, 100, 2500), 100) == 256);
  EXPECT(width(uniform(2000, 20, 2000), 20) == 256);
  // mixed sizes
  const BatchCall m24 = mixed(24, 10, 60), m350 = mixed(350, 10, 60), m4096 = mixed(4096, 10, 60);
  EXPECT(width(m24, 100) == 512 && width(m24, 40) == 512 && width(mixed(200, 10, 60), 100) == 512);
  EXPECT(width(m350, 100) == 256 && width(m350, 40) == 256 && width(m4096, 100) == 256 && width(m4096, 50) == 256);
  EXPECT(width(mixed(350, 4, 30), 50) == 256 && width(mixed(1000, 4, 30), 50) == 128);
  // LPs of other paths change nothing: 24 small ones among 3000 too large, or empty
  BatchCall few = mixed(24, 10, 60);
  for (int i = 0; i < 3000; ++i) few.add(129 + i, 5000), few.add(5, 0);
  EXPECT(few.lps == 24 && few.max_cols == m24.max_cols && few.cols == m24.cols && width(few, 100) == 512);
  // autotuned choices stay with the LPs per SM they were timed at
  sov::TunedWidths tuned;
  tuned.set(128, sov::lps_per_sm(148, 4096), {256, 1});
  EXPECT(tuned.find(128, sov::lps_per_sm(148, 3072)).threads == 256 && tuned.find(128, sov::lps_per_sm(148, 593)).per_sm == 1);
  for (int lps : {1, 24, 148, 149, 296, 297, 444, 445, 592}) EXPECT(tuned.find(128, sov::lps_per_sm(148, lps)).threads == 0);
  EXPECT(tuned.find(96, sov::lps_per_sm(148, 4096)).threads == 0);
  tuned.set(128, sov::lps_per_sm(148, 24), {512, 0});
  EXPECT(tuned.find(128, 1).threads == 512 && tuned.find(128, 5).threads == 256 && sov::lps_per_sm(148, 0) == 1);
  std::printf("failures %d\n", failures);
  return failures != 0;
}
