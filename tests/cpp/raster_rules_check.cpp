// Checks the tile rasteriser's shortcuts (gbr_math.h) against what they stand
// for: walk_first_late_row against walk_row_late over every width <= W, top
// row < H and row (a row before it must not be late), and box_bounds against
// depth_at and edge_inside at every pixel of random triangles' boxes; tight_box
// and row_span against edge_inside at the pixels of their bbox4; ssao_tap against ssao_count
// wherever ssao_exact holds; shadow_bias below kBiasFullCos; and shadow_limits
// and depth_below against the tests they stand for; and the two-part 1 / 255 and
// 1 / 350000.
// Usage: raster_rules_check W H <random boxes>; exit code 0 when all hold.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "gbr_shade_math.h"

using namespace gbr;

int main(int argc, char** argv) {
  if (argc < 4) return 2;
  const int W = atoi(argv[1]), H = atoi(argv[2]), n = atoi(argv[3]);
  long early = 0, late = 0;
#pragma omp parallel for schedule(dynamic, 8) reduction(+ : early, late)
  for (int w = 1; w <= W; w++)
    for (int miny = 0; miny < H; miny++) {
      const float iw = 1.0f / (float)w, fm = (float)miny;  // walk_row_late's arithmetic, 1 / w hoisted
      for (int r = 0; r <= H - miny; r++) {
        const bool l = floorf(fmaf((float)(r * w), iw, fm)) != fm + (float)r;
        early += l && r < walk_first_late_row(miny);
        late += l;
      }
    }
  std::mt19937 rng(5);
  auto uni = [&](float a, float b) { return std::uniform_real_distribution<float>(a, b)(rng); };
  long bad = 0, full = 0, bounded = 0;
  for (int i = 0; i < n; i++) {
    // vertices from sub-pixel to far off screen, near, far and mixed depths, some degenerate
    const float span = powf(10.0f, uni(-0.5f, 5.0f));
    float x[3], y[3], z[3];
    const float z0 = powf(10.0f, uni(1.31f, 5.54f));
    for (int k = 0; k < 3; k++) {
      x[k] = roundf(uni(-span, span) + 800.0f);
      y[k] = roundf(uni(-span, span) + 500.0f);
      z[k] = (rng() & 3) ? z0 : powf(10.0f, uni(1.31f, 5.54f));
    }
    if (!(rng() & 15)) x[2] = x[1], y[2] = y[1];
    const f3 xv = mk3(x[0], x[1], x[2]), yv = mk3(y[0], y[1], y[2]);
    const f3 dv = mk3(rcp(fdiv(z[0], kDepthFar)), rcp(fdiv(z[1], kDepthFar)), rcp(fdiv(z[2], kDepthFar)));
    float A, B, C;
    plane_const(dv, xv, yv, rconstant(xv, yv), &A, &B, &C);
    const EdgeTest e = make_edge(x[0], y[0], x[1], y[1], x[2], y[2]);
    const int x0 = (int)(rng() % 1600), y0 = (int)(rng() % 1000), x1 = x0 + (int)(rng() % 16), y1 = y0 + (int)(rng() % 16);
    uint32_t lo, hi;
    const bool f = box_bounds(A, B, C, e, x0, y0, x1, y1, &lo, &hi);
    full += f;
    bounded += lo != 0;
    for (int py = y0; py <= y1; py++)
      for (int px = x0; px <= x1; px++) {
        const uint32_t d = depth_at(A, B, C, (float)px, (float)py);
        if (d < lo || d > hi || (f && !edge_inside(e, (float)px, (float)py))) bad++;
      }
  }
  long tight = 0, empty = 0, outside = 0, spans = 0;
  const float sizes[5][2] = {{3840, 2160}, {1024, 1024}, {1920, 1080}, {64, 48}, {17, 9}};
  for (int i = 0; i < n; i++) {
    const float w = sizes[i % 5][0], h = sizes[i % 5][1];
    // around the surface and its far corner, extents from sub-pixel to over 64, some collinear
    const float span = powf(10.0f, uni(-0.5f, 3.0f)), cx = (i & 8) ? w : uni(0, w), cy = (i & 8) ? h : uni(0, h);
    f3 p[3];
    for (int k = 0; k < 3; k++) p[k] = mk3(cx + uni(-span, span), cy + uni(-span, span), 100.0f);
    if (!(rng() & 7)) p[2] = mk3(p[0].x + 2.0f * (p[1].x - p[0].x), p[0].y + 2.0f * (p[1].y - p[0].y), 100.0f);
    if (!(rng() & 63)) p[1].x = NAN;
    float mm[4], tm[4];
    bbox4(p[0], p[1], p[2], w, h, mm);
    for (int k = 0; k < 4; k++) tm[k] = mm[k];
    const f3 xv = mk3(roundf(p[0].x), roundf(p[1].x), roundf(p[2].x));
    const f3 yv = mk3(roundf(p[0].y), roundf(p[1].y), roundf(p[2].y));
    const int kind = tight_box(xv, yv, w, h, tm);
    tight += kind == kBoxTight;
    empty += kind == kBoxEmpty;
    EdgeTest e = make_edge(xv.x, yv.x, xv.y, yv.y, xv.z, yv.z);
    if (on_surface(xv, yv, w, h)) {  // the spans of rows, 16 columns at a time from a column near the triangle
      EdgeTest f = e;
      f.s0 *= e.sign, f.sa *= e.sign, f.sb *= e.sign, f.t0 *= e.sign, f.ta *= e.sign, f.tb *= e.sign;
      const float tx = 16.0f * floorf(uni(mm[0], mm[1]) / 16.0f);
      for (float py = mm[2]; py < mm[3]; py += (mm[3] - mm[2] > 80 ? 7 : 1)) {
        int xa = 0, xb = 15;
        row_span((f.s0 + f.sb * py) + f.sa * tx, (f.t0 + f.tb * py) + f.ta * tx, f.bound, span_slope(f.sa),
                 span_slope(f.ta), span_slope(-(f.sa + f.ta)), kind != kBoxAny, &xa, &xb);
        spans += xa > 0 || xb < 15;
        for (int k = 0; k < 16; k++)
          if ((k < xa || k > xb) && edge_inside(e, tx + (float)k, py)) outside++;
      }
    }
    if (kind == kBoxAny) continue;
    for (float py = mm[2]; py < mm[3]; py++)
      for (float px = mm[0]; px < mm[1]; px++) {
        const bool in = px >= tm[0] && px < tm[1] && py >= tm[2] && py < tm[3];
        if ((!in || kind == kBoxEmpty) && edge_inside(e, px, py)) outside++;
      }
  }
  printf("tight=%ld empty=%ld spans=%ld outside=%ld\n", tight, empty, spans, outside);
  bad += outside;
  long taps = 0, inexact = 0, wrong = 0;
  for (int i = 0; i < n; i++) {
    // distances over the whole range, every other one within 3 units of a power of two
    float dep = powf(2.0f, uni(-1.0f, 18.42f));
    if (i & 1) dep = exp2f((float)(3 + rng() % 16)) + uni(-3.0f, 3.0f);
    const uint32_t d0 = f2u_sat(dep / kDepthFar * kMulInt);
    dep = depth_to_dist(d0);
    if (!ssao_exact(dep)) {
      inexact++;
      continue;
    }
    const float t[5] = {(dep + -2.0f) * kTwo32, (dep + -1.0f) * kTwo32, dep * kTwo32, (dep + 1.0f) * kTwo32,
                        (dep + 2.0f) * kTwo32};
    for (int k = 0; k < 40; k++) {
      uint32_t d = rng();
      if (k < 36) {  // at and around every threshold
        const float at = t[k % 5] / kDepthFar;
        d = f2u_sat(at) + (uint32_t)((int)(rng() % 5) - 2) * ((k & 8) ? 1u : 300u);
      }
      if (k == 36) d = 0;
      if (k == 37) d = kDepthClear;
      taps++;
      wrong += ssao_tap(d, (2.0f - dep) * 0.125f) - kSsaoTapZero !=
               (uint32_t)ssao_count(depth_scaled(d), t[0], t[1], t[2], t[3], t[4]);
    }
  }
  // every cosine up to kBiasFullCos has the full bias
  long cosines = 0;
  for (float c = 0.05f; c <= kBiasFullCos; c = nextafterf(c, 2.0f)) cosines += shadow_bias(c) != kShadowBias;
  long shadow = 0;
  for (int i = 0; i < n; i++) {
    const float dpth = (i & 3) ? powf(10.0f, uni(-3.0f, 5.54f)) : uni(0.0f, 120.0f), bias = uni(5.0f, 50.0f);
    uint32_t lo, hi;
    if (!shadow_limits(dpth, bias, &lo, &hi)) continue;
    for (int k = 0; k < 24; k++) {
      const uint32_t near = (k & 1) ? lo : hi, step = 1u << (rng() % 12);
      uint32_t d = (k & 2) ? near + rng() % step : near - rng() % step;
      if (k == 20) d = 0;
      if (k == 21) d = kDepthClear;
      if (k > 21) d = rng();
      const bool t = dpth > depth_to_dist(d) + bias;
      shadow += (d < lo && !t) || (d > hi && t);
    }
  }
  for (int i = 0; i < n; i++) {  // the limit, and the depths on either side of it
    const float t = (i & 7) ? powf(10.0f, uni(-5.0f, 5.6f)) : uni(-10.0f, 10.0f);
    const uint32_t d = depth_below(t);
    shadow += (d > 0 && !(depth_to_dist(d - 1) < t)) || (d < kDepthClear && depth_to_dist(d) < t);
  }
  for (int c = 0; c < 256; c++)
    shadow += fma_((float)c, kInv255Hi, (float)c * kInv255Lo) != fdiv((float)c, 255.0f);
  // over_far for every depth of its range
  for (float z = 1e-6f; z <= 1e12f; z = nextafterf(z, 1e30f)) shadow += over_far(z) != fdiv(z, kDepthFar);
  printf("cosines=%ld shadow=%ld\n", cosines, shadow);
  bad += cosines + shadow;
  printf("taps=%ld inexact=%ld wrong=%ld\n", taps, inexact, wrong);
  bad += wrong;
  printf("early=%ld late=%ld boxes=%d full=%ld bounded=%ld bad=%ld\n", early, late, n, full, bounded, bad);
  return early == 0 && late > 0 && bad == 0 && tight > 0 && empty > 0 && spans > 0 && taps > 0 && inexact > 0 && full > 0 && bounded > 0 ? 0 : 1;
}
