// Checks walk_skip_rows (gbr_math.h, what the rasterisers apply: bits of up to
// 32 rows, stepped) against walk_visits at every row, over windows of 16 rows
// (the tiles) and the two windows of up to 32 that a cube face's small box
// takes.  Usage: walk_skip_check <seed> <random boxes>; exit code 0 when all hold.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "gbr_math.h"

using namespace gbr;

static long bad = 0, skipped = 0;

static void check(int minx, int w, int miny, int h, int y0, int y1, int ty, int chunk) {
  const uint32_t xr = (uint32_t)minx | ((uint32_t)(minx + w) << 16), yr = (uint32_t)miny | ((uint32_t)(miny + h) << 16);
  uint32_t want = 0;
  for (int py = y0; py < y1; py++)
    if (!walk_visits(0, py - miny, w, h, (float)miny, chunk)) want |= 1u << (py - ty);
  skipped += __builtin_popcount(want);
  if (walk_skip_rows(xr, yr, y0, y1, ty, chunk) != want && bad++ < 5)
    std::printf("w=%d h=%d miny=%d rows [%d, %d) chunk=%d\n", w, h, miny, y0, y1, chunk);
}

static void box(int minx, int w, int miny, int h) {
  for (int chunk : {500, 300}) {
    for (int ty = miny & ~15; ty < miny + h; ty += 16)
      check(minx, w, miny, h, std::max(miny, ty), std::min(miny + h, ty + 16), ty, chunk);
    if (w * h <= 64) {
      check(minx, w, miny, h, miny, std::min(miny + h, miny + 32), miny, chunk);
      if (h > 32) check(minx, w, miny, h, miny + 32, miny + h, miny + 32, chunk);
    }
  }
}

int main(int argc, char** argv) {
  std::mt19937 rng(argc > 1 ? (unsigned)atoi(argv[1]) : 1);
  const int n = argc > 2 ? atoi(argv[2]) : 1000;
  for (int w = 1; w <= 700; w++)  // across both chunk sizes, and all small boxes of a face
    for (int miny : {0, 1, 2, 5, 11, 30, 200})
      for (int h : {1, 2, 3, 16, 17, 33, 40, 64, 500}) box(w % 7, w, miny, h);
  for (int i = 0; i < n; i++) {
    const int w = 1 + (int)(rng() % 3840), miny = (int)(rng() % ((i & 1) ? 2159 : 40));
    box((int)(rng() % (3841 - w)), w, miny, 1 + (int)(rng() % (2160 - miny)));
  }
  std::printf("skipped=%ld bad=%ld\n", skipped, bad);
  return bad == 0 && skipped > 0 ? 0 : 1;
}
