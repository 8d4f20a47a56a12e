// gbr_shade_math.h — scalar pieces of kernel3 and the post passes that stand
// for longer expressions of the reference, shared with their host checks.
#pragma once

#include "gbr_math.h"

namespace gbr {

// (float)d / 2^32 * 350000: the division by 2^32 only shifts the exponent
// (no rounding, no underflow for d >= 1), so it is a multiplication by 2^-32.
constexpr float kInvMulInt = 2.3283064365386963e-10f;
GBR_HD float depth_to_dist(uint32_t d) { return ((float)d * kInvMulInt) * kDepthFar; }

// depth_to_dist(d) compared with a threshold t: (float)d * 2^-32 is exact and
// a scaling by a power of two commutes with rounding (every value here is a
// normal float), so depth_to_dist(d) = RN((float)d * 350000) * 2^-32, and
// depth_to_dist(d) > t exactly when RN((float)d * 350000) > t * 2^32.
constexpr float kTwo32 = 4294967296.0f;
GBR_HD float depth_scaled(uint32_t d) { return (float)d * kDepthFar; }

// The smallest d with depth_to_dist(d) >= t (UINT_MAX if there is none below
// it): depth_to_dist(d) < t is d < depth_below(t), since depth_to_dist does
// not decrease.  Bisected from a bracket 10 * 2^-24 of t wide to either side.
GBR_HD uint32_t depth_below(float t) {
  if (!(t > 0.0f)) return 0u;
  const float slack = t * 6e-7f;
  uint32_t lo = f2u_sat((t - slack) * (kMulInt / kDepthFar)), hi = f2u_sat((t + slack) * (kMulInt / kDepthFar));
  hi += hi != 0xFFFFFFFFu;
  while (lo < hi) {  // below lo: less than t; hi and above: not (or the end)
    const uint32_t mid = lo + (hi - lo) / 2;
    if (depth_to_dist(mid) < t)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// 1 / 255 = kInv255Hi + kInv255Lo: fma(x, hi, x * lo) is fdiv(x, 255.0f) for
// every byte x (tests/cpp/raster_rules_check.cpp).
constexpr float kInv255Hi = 0x1.010102p-8f, kInv255Lo = -0x1.fdfdfep-33f;

// How many of the thresholds t0 < t1 < t2 < t3 < t4 lie below d2, i.e.
// (d2 > t0) + ... + (d2 > t4): the thresholds dep + z (z = -2..2, dep <=
// 350000) are strictly increasing in float, so the predicates are monotone and
// three comparisons find the count.
GBR_HD int ssao_count(float d2, float t0, float t1, float t2, float t3, float t4) {
  return d2 > t2 ? (d2 > t4 ? 5 : (d2 > t3 ? 4 : 3)) : (d2 > t1 ? 2 : (d2 > t0 ? 1 : 0));
}

// ssao_count of one tap for a pixel at distance dep (ssao_exact), given c8 =
// (2 - dep) / 8: how many of dep + k, k = -2..2, lie below the tap's distance
// v.  That is ceil(v - dep + 2) clamped to 0..5, and u = (v - dep + 2) / 8 is
// one fused operation, exact wherever it falls inside (0, 1) (v and dep are
// then within a factor of two and share their grid): clamped by saturation,
// multiplied back and rounded up to an integer by the addition of 1.5 * 2^23.
// Returns that float's bits, kSsaoTapZero + count: six instructions and no
// compare or select per tap.
constexpr uint32_t kSsaoTapZero = 0x4B400000u;
GBR_HD uint32_t ssao_tap(uint32_t d, float c8) {
  const float u = fma_(depth_scaled(d), kInvMulInt * 0.125f, c8);
#if defined(__CUDA_ARCH__)
  return __float_as_uint(fminf(__fmaf_ru(__saturatef(u), 8.0f, 12582912.0f), 12582917.0f));
#else
  return kSsaoTapZero + (uint32_t)fminf(ceilf(clampf_(u, 0.0f, 1.0f) * 8.0f), 5.0f);
#endif
}
// Are the thresholds dep + k exact?  Below dep always (dep >= 8); above it
// unless dep + k crosses into a binade that cannot hold it.
GBR_HD bool ssao_exact(float dep) {
  return dep >= 8.0f && (dep + 1.0f) - dep == 1.0f && (dep + 2.0f) - dep == 2.0f;
}

// The shadow bias of generate_hard_occlusion for a cosine of incidence (cl2.cl:2604-2608).
GBR_HD float shadow_bias(float cosine) {
  const float acos_res = rational_acos(clampf_(cosine, 0.05f, 0.95f));
  return clampf_(kShadowBias * gbr_tanf(acos_res), 0.1f * kShadowBias, kShadowBias);
}
// shadow_bias is kShadowBias for every cosine up to this one (checked for
// every float of its range): beyond 45 degrees the tangent exceeds 1.
constexpr float kBiasFullCos = 0.70f;

// Limits of a shadow tap's test dpth > depth_to_dist(d) + bias (bias at most
// 50): true for every d < *lo, false for every d > *hi.  The limit is dpth -
// bias in depth units; 10 * 2^-24 of dpth to either side cover the at most 7
// roundings of the two forms.  Returns false where the limit is near the end
// of the range and says nothing.
GBR_HD bool shadow_limits(float dpth, float bias, uint32_t* lo, uint32_t* hi) {
  const float lim = dpth - bias, slack = dpth * 6e-7f;
  *lo = f2u_sat((lim - slack) * (kMulInt / kDepthFar));
  *hi = f2u_sat((lim + slack) * (kMulInt / kDepthFar));
  return lim < 349000.0f;
}

}  // namespace gbr
