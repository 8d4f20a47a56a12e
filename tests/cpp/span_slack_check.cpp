// Checks row_span_slack with span_slack (gbr_math.h) against edge_inside: for
// records with vertices off the surface but near_surface, no pixel of a tile row
// outside the span may be covered.  Usage: span_slack_check <seed> <triangles>;
// exit code 0 when all hold and most rows are narrowed.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "gbr_math.h"

using namespace gbr;

int main(int argc, char** argv) {
  std::mt19937 rng(argc > 1 ? (unsigned)atoi(argv[1]) : 1);
  const int n = argc > 2 ? atoi(argv[2]) : 100000;
  auto uni = [&](float a, float b) { return std::uniform_real_distribution<float>(a, b)(rng); };
  const float sizes[5][2] = {{3840, 2160}, {1024, 1024}, {1920, 1080}, {64, 48}, {17, 9}};
  long outside = 0, rows = 0, narrowed = 0, used = 0, covered = 0;
  for (int i = 0; i < n; i++) {
    const float w = sizes[i % 5][0], h = sizes[i % 5][1];
    f3 p[3];
    // an edge of any slope through the surface, vertices up to 2^18 away, some
    // thin, some collinear, some with a vertex on the surface
    const float far = powf(10.0f, uni(0.5f, 5.4f));
    const float cx = uni(0, w), cy = uni(0, h), a = uni(0, 6.2831853f);
    for (int k = 0; k < 3; k++) {
      const float d = uni(-far, far), thin = (i & 3) ? uni(-far, far) : uni(-3, 3);
      p[k] = mk3(roundf(cx + d * cosf(a) - thin * sinf(a)), roundf(cy + d * sinf(a) + thin * cosf(a)), 100.0f);
    }
    if (!(rng() & 3)) p[rng() % 3] = mk3(roundf(uni(0, w)), roundf(uni(0, h)), 100.0f);
    if (!(rng() & 15)) p[2] = mk3(2 * p[1].x - p[0].x, 2 * p[1].y - p[0].y, 100.0f);
    if (!(rng() & 255)) p[rng() % 3].x = (rng() & 1) ? NAN : INFINITY;
    const f3 xv = mk3(p[0].x, p[1].x, p[2].x), yv = mk3(p[0].y, p[1].y, p[2].y);
    if (on_surface(xv, yv, w, h) || !near_surface(xv, yv)) continue;
    used++;
    const EdgeTest e = make_edge(xv.x, yv.x, xv.y, yv.y, xv.z, yv.z);
    EdgeTest f = e;  // the records' form: the sign folded in
    f.s0 *= e.sign, f.sa *= e.sign, f.sb *= e.sign, f.t0 *= e.sign, f.ta *= e.sign, f.tb *= e.sign;
    for (int k = 0; k < 24; k++) {
      // tiles on an edge, where one crosses the surface, and anywhere
      float tx = 16.0f * floorf(uni(0, w) / 16.0f), py = floorf(uni(0, h));
      if (k & 1) {
        const int u = (int)(rng() % 3), v = (u + 1) % 3;
        const float q = uni(0, 1), x = p[u].x + q * (p[v].x - p[u].x), y = p[u].y + q * (p[v].y - p[u].y);
        if (!(x >= 0 && x < w && y >= 0 && y < h)) continue;
        tx = 16.0f * floorf(x / 16.0f), py = floorf(y);
      }
      int xa = 0, xb = 15;
      const float slack = span_slack(f.s0, f.sa, f.sb, f.t0, f.ta, f.tb, f.bound, tx + 16.0f, py);
      row_span_slack((f.s0 + f.sb * py) + f.sa * tx, (f.t0 + f.tb * py) + f.ta * tx, f.bound, span_slope(f.sa),
                     span_slope(f.ta), span_slope(-(f.sa + f.ta)), slack, slack, &xa, &xb);
      rows++;
      narrowed += xa > 0 || xb < 15;
      for (int c = 0; c < 16; c++)
        if (edge_inside(e, tx + (float)c, py)) {
          covered++;
          outside += c < xa || c > xb;
        }
    }
  }
  std::printf("used=%ld rows=%ld narrowed=%ld covered=%ld outside=%ld\n", used, rows, narrowed, covered, outside);
  return outside == 0 && used > n / 4 && narrowed > rows / 4 && covered > 0 ? 0 : 1;
}
