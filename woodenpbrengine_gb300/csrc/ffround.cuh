// ffround.cuh — double expressions rounded to float, evaluated in pairs of
// floats on the device.
//
// The reference writes several of its expressions in double (every PI, the
// sphere quadratic, the square roots of 1 - x^2) and rounds the result to
// float. GB300 issues one FP64 instruction per 16 cycles and SM where it
// issues four FP32 ones per cycle, and those expressions kept the FP64 pipe
// 73 % busy in the spawn kernel of a 1080p frame, 75 % in the shadow traversal
// of a sphere scene and 41 to 49 % in the differentiable estimator's. Here
// each one is evaluated as an unevaluated sum hi + lo of two floats
// (error-free products by fused multiply-add, error-free sums by Knuth's
// TwoSum; T. J. Dekker, "A floating-point technique for extending the
// available precision", Numer. Math. 18, 1971) with a relative error below
// 2^-43, and the float result is taken only if every number within 2^-42 of
// hi + lo rounds to the same float (Ziv's rounding test). The double
// expressions lie within 2^-50 of the exact value (tr_rcp's, of six roundings,
// within 2^-50.4; the others within 2^-51), so they then round to that float
// too: the result is the double expression's, bit for bit. Everything else
// (about one operand in 10^5, and operands so large, small or special that an
// error term could leave the float range) takes the double expression itself,
// out of line.
//
// Per pass, before -> after: 1080p full frame, spawn 171 -> 143 us, finish 70
// -> 57 us; textured spheres at 1080p, shadow rays 144 -> 112 us; 512 x 512
// differentiable pass, spawn 47 -> 42 us, shadow rays 46 -> 33 us.
#pragma once

#include <stdint.h>

#include "wpbr_fmath.h"

#if defined(__CUDACC__)
#define WPBR_HD_SLOW __host__ __device__ __noinline__ inline
#else
#define WPBR_HD_SLOW __attribute__((noinline)) inline
#endif

namespace wpbr {

namespace ff {

WPBR_HD float fma_(float a, float b, float c) {
#if defined(__CUDA_ARCH__)
  return __fmaf_rn(a, b, c);
#else
  return __builtin_fmaf(a, b, c);
#endif
}
// 1 / x and 1 / sqrt(x) within a few units in the last place: starting values
// and correction factors, never results. WPBR_FF_PERTURB (a test) moves the
// host's values away from the true ones by that many units.
WPBR_HD float rcp_approx(float x) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#elif defined(WPBR_FF_PERTURB)
  return wpbr_fm::u2f(wpbr_fm::f2u(1.0f / x) + WPBR_FF_PERTURB);
#else
  return 1.0f / x;
#endif
}
WPBR_HD float rsqrt_approx(float x) {
#if defined(__CUDA_ARCH__)
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#elif defined(WPBR_FF_PERTURB)
  return wpbr_fm::u2f(wpbr_fm::f2u(1.0f / __builtin_sqrtf(x)) + WPBR_FF_PERTURB);
#else
  return 1.0f / __builtin_sqrtf(x);
#endif
}

struct FF {
  float h, l;
};
constexpr float kTiny = 0x1p-40f, kHuge = 0x1p40f;  // operands' range: no error term underflows, nothing overflows
constexpr float kMargin = 0x1p-42f;                 // accepted relative distance to the exact value

// |x| in [kTiny, kHuge] (false for NaN)
WPBR_HD bool in_range(float x) {
  const float a = wpbr_fm::fabs_(x);
  return a >= kTiny && a <= kHuge;
}
// a + b exactly, |a| >= |b| or a = 0
WPBR_HD FF fast_two_sum(float a, float b) {
  const float s = a + b;
  return FF{s, b - (s - a)};
}
WPBR_HD FF two_sum(float a, float b) {
  const float s = a + b;
  const float t = s - a;
  return FF{s, (a - (s - t)) + (b - t)};
}
WPBR_HD FF two_prod(float a, float b) {
  const float p = a * b;
  return FF{p, fma_(a, b, -p)};
}
// (h + l) * f, relative error below 2^-46
WPBR_HD FF mul_f(FF a, float f) {
  const float p = a.h * f;
  const float e = fma_(a.l, f, fma_(a.h, f, -p));
  return fast_two_sum(p, e);
}
// sqrt(h + l) for h in range: the residual of the rounded root gives the next 24 bits
WPBR_HD FF sqrt_ff(FF a) {
  const float s = wpbr_fm::sqrt_(a.h);
  const float r = fma_(-s, s, a.h) + a.l;
  return FF{s, r * (0.5f * rsqrt_approx(a.h))};
}
// (nh + nl) / (dh + dl), one correction step of an approximate quotient
WPBR_HD FF div_ff(FF n, FF d) {
  const float y = rcp_approx(d.h);
  const float q = n.h * y;
  const float r = fma_(-q, d.l, fma_(-q, d.h, n.h) + n.l);
  return fast_two_sum(q, r * y);
}
// The float that everything within kMargin of h + l rounds to; false when
// there is none (|l| is at most about half a unit of h).
WPBR_HD bool round_ff(FF a, float* out) {
  const float lo = a.h + fma_(-kMargin, a.h, a.l);
  const float hi = a.h + fma_(kMargin, a.h, a.l);
  *out = lo;
  return lo == hi;
}

}  // namespace ff

// The double constants of the reference's expressions as float pairs (48 of
// their 53 bits: a relative error below 2^-48).
struct FFConst {
  double d;
  float h, l;
};
constexpr FFConst ff_const(double d) { return FFConst{d, (float)d, (float)(d - (double)(float)d)}; }

// (float)((double)x * C)
WPBR_HD_SLOW float mul_const_d(float x, double c) { return (float)((double)x * c); }
WPBR_HD float mul_const(float x, FFConst c) {
#if defined(__CUDA_ARCH__) || defined(WPBR_FF_HOST)
  float r;
  if (ff::in_range(x) && ff::round_ff(ff::mul_f(ff::FF{c.h, c.l}, x), &r)) return r;
  if (x == 0.0f) return x;  // C is positive
#endif
  return mul_const_d(x, c.d);
}
// (float)((double)x / C): times the reciprocal, given as a pair
struct FFRecip {
  double d;     // C
  float h, l;   // 1 / C
};
constexpr FFRecip ff_recip(double d) { return FFRecip{d, (float)(1.0 / d), (float)(1.0 / d - (double)(float)(1.0 / d))}; }
WPBR_HD_SLOW float div_const_d(float x, double c) { return (float)((double)x / c); }
WPBR_HD float div_const(float x, FFRecip c) {
#if defined(__CUDA_ARCH__) || defined(WPBR_FF_HOST)
  float r;
  if (ff::in_range(x) && ff::round_ff(ff::mul_f(ff::FF{c.h, c.l}, x), &r)) return r;
  if (x == 0.0f) return x;  // C is positive
#endif
  return div_const_d(x, c.d);
}

// (float)sqrt(max(0, 1.0 - (double)x)), the maximum as std::max(0.0, .)
WPBR_HD_SLOW float sqrt_one_minus_d(float x) {
  const double a = 1.0 - (double)x;
  return (float)wpbr_fm::sqrt_d(0.0 > a ? 0.0 : a);
}
WPBR_HD float sqrt_one_minus(float x) {
#if defined(__CUDA_ARCH__) || defined(WPBR_FF_HOST)
  if (x >= 1.0f) return 0.0f;
  if (x >= 0.0f) {
    const float h = 1.0f - x;  // at least 2^-24
    float r;
    if (ff::round_ff(ff::sqrt_ff(ff::FF{h, (1.0f - h) - x}), &r)) return r;
  }
#endif
  return sqrt_one_minus_d(x);
}

// (float)((double)u * (1.0 - (double)c) + (double)c)
WPBR_HD_SLOW float lerp_to_one_d(float u, float c) { return (float)((double)u * (1.0 - (double)c) + (double)c); }
WPBR_HD float lerp_to_one(float u, float c) {
#if defined(__CUDA_ARCH__) || defined(WPBR_FF_HOST)
  if (u >= 0x1p-30f && u <= 1.0f && c >= 0x1p-30f && c < 1.0f) {
    const float h = 1.0f - c;
    const ff::FF t = ff::mul_f(ff::FF{h, (1.0f - h) - c}, u);
    const ff::FF s = ff::two_sum(t.h, c);
    float r;
    if (ff::round_ff(ff::fast_two_sum(s.h, s.l + t.l), &r)) return r;
  }
#endif
  return lerp_to_one_d(u, c);
}

// (float)(1.0 / (((((C * ax) * ay) * c4) * g) * g)) in double (Trowbridge-Reitz D)
WPBR_HD_SLOW float tr_rcp_d(double c, float ax, float ay, float c4, float g) {
  const double den = ((((c * (double)ax) * (double)ay) * (double)c4) * (double)g) * (double)g;
  return (float)(1.0 / den);
}
WPBR_HD float tr_rcp(FFConst c, float ax, float ay, float c4, float g) {
#if defined(__CUDA_ARCH__) || defined(WPBR_FF_HOST)
  // the partial products stay in [2^-68, 2^100] and the denominator that is
  // inverted below 2^70, so no error term is lost to underflow
  if (ax >= 0x1p-16f && ax <= 0x1p10f && ay >= 0x1p-16f && ay <= 0x1p10f && c4 >= 0x1p-30f && c4 <= 0x1p4f &&
      g >= 0x1p-4f && g <= 0x1p36f) {
    ff::FF d = ff::mul_f(ff::FF{c.h, c.l}, ax);
    d = ff::mul_f(d, ay);
    d = ff::mul_f(d, c4);
    d = ff::mul_f(d, g);
    d = ff::mul_f(d, g);
    float r;
    if (d.h <= 0x1p70f && ff::round_ff(ff::div_ff(ff::FF{1.0f, 0.0f}, d), &r)) return r;
  }
#endif
  return tr_rcp_d(c.d, ax, ay, c4, g);
}

// (float)((double)n / (C * (double)s))
WPBR_HD_SLOW float div_by_scaled_d(float n, double c, float s) { return (float)((double)n / (c * (double)s)); }
WPBR_HD float div_by_scaled(float n, FFConst c, float s) {
#if defined(__CUDA_ARCH__) || defined(WPBR_FF_HOST)
  if (ff::in_range(n) && ff::in_range(s)) {
    float r;
    if (ff::round_ff(ff::div_ff(ff::FF{n, 0.0f}, ff::mul_f(ff::FF{c.h, c.l}, s)), &r)) return r;
  } else if (n == 0.0f && ff::in_range(s)) {
    return n / s;  // a signed zero (C is positive)
  }
#endif
  return div_by_scaled_d(n, c.d, s);
}

// pbrt-v3's Quadratic as WoodenMath's getRootsQuadraticEquation is restated
// here: discriminant, root and q in double, the roots rounded to float and
// sorted.
struct Roots {
  float t0, t1;
  bool real;
};
WPBR_HD_SLOW Roots quadratic_d(float a, float b, float c) {
  double discrim = (double)b * (double)b - 4.0 * (double)a * (double)c;
  if (discrim < 0.0) return Roots{0.0f, 0.0f, false};
  double root = wpbr_fm::sqrt_d(discrim);
  double q = (b < 0.0f) ? -0.5 * ((double)b - root) : -0.5 * ((double)b + root);
  float r0 = (float)(q / (double)a);
  float r1 = (float)((double)c / q);
  return r0 > r1 ? Roots{r1, r0, true} : Roots{r0, r1, true};
}
WPBR_HD bool quadratic(float a, float b, float c, float* t0, float* t1) {
#if defined(__CUDA_ARCH__) || defined(WPBR_FF_HOST)
  const float aa = wpbr_fm::fabs_(a), ab = wpbr_fm::fabs_(b), ac = wpbr_fm::fabs_(c);
  constexpr float kLo = 0x1p-24f, kHi = 0x1p24f;
  if (aa >= kLo && aa <= kHi && ab >= kLo && ab <= kHi && ac >= kLo && ac <= kHi) {
    // b^2 - 4ac: both products as exact pairs, their difference
    // s.h + (s.l + (e.h + e.l)) with s.l = 0 whenever much cancels
    const ff::FF p = ff::two_prod(b, b), m = ff::two_prod(4.0f * a, c);
    const ff::FF s = ff::two_sum(p.h, -m.h);
    const ff::FF e = ff::two_sum(p.l, -m.l);
    const ff::FF v = ff::two_sum(s.h, e.h);
    const ff::FF d = ff::fast_two_sum(v.h, s.l + (v.l + e.l));
    // the roundings of the low part are below 2^-45 of the discriminant when
    // |e.h| is at most the discriminant and |s.l| at most 2^-22 of it, which
    // fails only within about 2^-23 of a tangent ray
    const float ah = wpbr_fm::fabs_(d.h);
    if (ah >= wpbr_fm::fabs_(e.h) && 0x1p-22f * ah >= wpbr_fm::fabs_(s.l) && ah >= 0x1p-60f) {
      if (d.h < 0.0f) return false;
      const ff::FF root = ff::sqrt_ff(d);
      const ff::FF w = ff::two_sum(ab, root.h);
      ff::FF q = ff::fast_two_sum(w.h, w.l + root.l);  // |b| + root; q = +-0.5 times it
      const float half = b < 0.0f ? 0.5f : -0.5f;
      q.h *= half;
      q.l *= half;
      float r0, r1;
      const bool ok0 = ff::round_ff(ff::div_ff(q, ff::FF{a, 0.0f}), &r0);
      const bool ok1 = ff::round_ff(ff::div_ff(ff::FF{c, 0.0f}, q), &r1);
      if (ok0 && ok1) {
        *t0 = r0 > r1 ? r1 : r0;
        *t1 = r0 > r1 ? r0 : r1;
        return true;
      }
    }
  }
#endif
  const Roots r = quadratic_d(a, b, c);
  *t0 = r.t0;
  *t1 = r.t1;
  return r.real;
}

}  // namespace wpbr
