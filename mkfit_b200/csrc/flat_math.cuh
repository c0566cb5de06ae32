// Elementary arithmetic for the Kalman step in two forms with one result but
// for the two rare roundings named below.
//
// ExactMath is the plain form: IEEE division and square root, double
// elementary functions rounded once to float (kalman.cuh f_*). Each of its
// roughly forty divisions and roots per fit step tests for its special cases and
// branches, and the double functions do too: about 190 of the step's 1900
// instructions, and a basic block ends at each, so nothing of one chain is
// issued while another waits.
//
// FlatMath computes the same values without a branch, for operands in a
// safe range, and keeps the smallest and largest operand it was given: when
// one lay outside (or was NaN), ok() is false and the caller repeats the step
// with ExactMath. Methods: quotient and root from an approximate reciprocal
// (root) by fused residuals (P. Markstein, IBM J. Res. Dev. 34, 1990),
// correctly rounded but for the reciprocal of a mantissa of all ones, which
// is one ulp off, and quotients by such a number (two of 2^26 tried); sine and cosine by their Taylor series after reduction by
// multiples of pi/2 in two parts; logarithm by the series of
// 2 artanh((m - 1) / (m + 1)). The double results are within a few 1e-16 of
// the exact value, so they round to ExactMath's float but where that value
// lies within ~1e-16 of a rounding boundary.
#pragma once

#include <cuda_runtime.h>

namespace mkfg {

__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Minimum / maximum that keep a NaN.
__device__ __forceinline__ float min_nan(float a, float b) {
  float y;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
  return y;
}
__device__ __forceinline__ float max_nan(float a, float b) {
  float y;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(y) : "f"(a), "f"(b));
  return y;
}

// 1 / b, a / b and sqrt(x) for normal operands (a may be 0) whose result is a
// normal finite number; an overflow gives NaN. ok() leaves the step's
// divisors and roots within [2^-80, 2^120].
__device__ __forceinline__ float flat_rcp(float b) {
  float y = rcp_approx(b);
  y = __fmaf_rn(__fmaf_rn(-b, y, 1.f), y, y);
  return __fmaf_rn(__fmaf_rn(-b, y, 1.f), y, y);
}
// a / b given y = flat_rcp(b).
__device__ __forceinline__ float flat_div_y(float a, float b, float y) {
  const float q = __fmul_rn(a, y);
  return __fmaf_rn(__fmaf_rn(-b, q, a), y, q);
}
__device__ __forceinline__ float flat_sqrt(float x) {
  const float y = rsqrt_approx(x);
  float g = __fmul_rn(x, y), h = __fmul_rn(0.5f, y);
  const float r = __fmaf_rn(-g, h, 0.5f);
  g = __fmaf_rn(g, r, g);
  h = __fmaf_rn(h, r, h);
  return __fmaf_rn(__fmaf_rn(-g, g, x), h, g);
}
// 1 / d in double from the float reciprocal: its error e ~ 2^-22 goes to
// e^3 in one step.
__device__ __forceinline__ double flat_rcp(double d) {
  const double y = rcp_approx((float)d);
  const double e = __fma_rn(-d, y, 1.0);
  return __fma_rn(__fma_rn(e, e, e), y, y);
}
// sqrt(s) in double from the float root.
__device__ __forceinline__ double flat_sqrt(double s) {
  const float f = (float)s;
  const float y = rsqrt_approx(f);
  const double h = 0.5f * y;
  double g = __fmul_rn(f, y);
  g = __fma_rn(__fma_rn(-g, g, s), h, g);
  return __fma_rn(__fma_rn(-g, g, s), h, g);
}

// sin and cos of x, |x| up to a few hundred.
__device__ __forceinline__ void flat_sincos(float x, float* s, float* c) {
  const float nf = rintf(x * 0.63661977f);  // 2 / pi
  const int n = (int)nf;
  const double N = nf;
  double r = __fma_rn(-N, 1.5707963267948966, (double)x);  // pi / 2, high part
  r = __fma_rn(-N, 6.123233995736766e-17, r);              // low part
  const double z = r * r;
  // Taylor coefficients 1 / 15!, -1 / 13!, ... ; |r| <= pi / 4.
  double p = -7.647163731819816e-13;
  p = __fma_rn(p, z, 1.6059043836821613e-10);
  p = __fma_rn(p, z, -2.505210838544172e-8);
  p = __fma_rn(p, z, 2.7557319223985893e-6);
  p = __fma_rn(p, z, -1.984126984126984e-4);
  p = __fma_rn(p, z, 8.333333333333333e-3);
  p = __fma_rn(p, z, -0.16666666666666666);
  const float sf = (float)__fma_rn(p * z, r, r);
  double q = 4.779477332387385e-14;
  q = __fma_rn(q, z, -1.1470745597729725e-11);
  q = __fma_rn(q, z, 2.08767569878681e-9);
  q = __fma_rn(q, z, -2.755731922398589e-7);
  q = __fma_rn(q, z, 2.48015873015873e-5);
  q = __fma_rn(q, z, -1.388888888888889e-3);
  q = __fma_rn(q, z, 4.1666666666666664e-2);
  q = __fma_rn(q, z, -0.5);
  const float cf = (float)__fma_rn(q, z, 1.0);
  const float a = n & 1 ? cf : sf, b = n & 1 ? sf : cf;
  *s = n & 2 ? -a : a;
  *c = (n + 1) & 2 ? -b : b;
}

// log(x), x a normal positive number: x = 2^e m with m in [sqrt(1/2), sqrt(2)).
__device__ __forceinline__ float flat_log(float x) {
  const int i = __float_as_int(x);
  const int e = (i - 0x3f3504f3) >> 23;
  const double m = __int_as_float(i - (e << 23));
  const double s = (m - 1.0) * flat_rcp(m + 1.0);
  const double z = s * s;
  double p = 1.0 / 19;
  p = __fma_rn(p, z, 1.0 / 17);
  p = __fma_rn(p, z, 1.0 / 15);
  p = __fma_rn(p, z, 1.0 / 13);
  p = __fma_rn(p, z, 1.0 / 11);
  p = __fma_rn(p, z, 1.0 / 9);
  p = __fma_rn(p, z, 1.0 / 7);
  p = __fma_rn(p, z, 1.0 / 5);
  p = __fma_rn(p, z, 1.0 / 3);
  const double t = 2.0 * s;
  return (float)__fma_rn((double)e, 0.6931471805599453, __fma_rn(t * z, p, t));
}

struct FlatMath {
  static constexpr bool kPlain = false;
  // Sizes of the operands seen: `lo`, `hi` those that bound others (momenta,
  // radii, sines; products of a few of them stay normal numbers), `wlo`,
  // `whi` those used on their own.
  float lo = 1.f, hi = 1.f, wlo = 1.f, whi = 1.f;
  __device__ __forceinline__ void see(float v) {
    lo = min_nan(lo, fabsf(v));
    hi = max_nan(hi, fabsf(v));
  }
  // A number that must be positive.
  __device__ __forceinline__ void see_wide(float v) {
    wlo = min_nan(wlo, v);
    whi = max_nan(whi, v);
  }
  // A dividend, or another number that only its size can spoil: a quotient
  // that overflows is NaN here and infinite there.
  __device__ __forceinline__ void see_top(float v) { hi = max_nan(hi, fabsf(v)); }
  __device__ __forceinline__ void see_angle(float v) { hi = max_nan(hi, fabsf(v) * 0x1p12f); }
  __device__ __forceinline__ bool ok() const {
    return lo >= 0x1p-20f && hi <= 0x1p20f && wlo >= 0x1p-90f && whi <= 0x1p90f;
  }
  // Operands already seen (or bounded by seen ones).
  __device__ __forceinline__ static float rcp(float b) { return flat_rcp(b); }
  __device__ __forceinline__ static float div(float a, float b) { return flat_div_y(a, b, flat_rcp(b)); }
  // a / b for a constant b, y the correctly rounded 1 / b.
  __device__ __forceinline__ static float div_const(float a, float b, float y) { return flat_div_y(a, b, y); }
  __device__ __forceinline__ static float sqrt(float x) { return flat_sqrt(x); }
  __device__ __forceinline__ void sincos(float x, float* s, float* c) {
    see_angle(x);
    flat_sincos(x, s, c);
  }
  __device__ __forceinline__ float log(float x) {
    see_wide(x);
    return flat_log(x);
  }
  // hypot_f of kalman.cuh.
  __device__ __forceinline__ float hypot(float x, float y) {
    const double dx = x, dy = y;
    const double s = dx * dx + dy * dy;
    see((float)s);
    return (float)flat_sqrt(s);
  }
  // (float)(1 / det).
  __device__ __forceinline__ float inv_det(double det) {
    const float f = (float)det;
    see_wide(fabsf(f));
    return (float)flat_rcp(det);
  }
};

}  // namespace mkfg
