// cr_math.cuh -- the correctly rounded value of DEPTH**(1.D0/3.D0), the
// Manning depth factor of rhs_dg_hydro.F, computed with IEEE-754 basic
// operations (+, -, *, /, fma, and the exact frexp / ldexp) and a
// single-precision logarithm whose error the method absorbs, so that the
// same source gives the same bits on the host and on the device.
//
// The exponent of the reference's expression is c = RN(1/3) = (1 - 2^-54)/3,
// the double nearest 1/3, so
//     x^c = x^(1/3) * x^(-2^-54/3) = cbrt(x) * (1 - 2^-54 ln(x) / 3 + O(2^-108 ln(x)^2)).
// cbrt(x) is formed to about 2^-100 relative accuracy as a double plus a
// correction term:
//   1. x = f 2^e (frexp), e = 3q + r with r in {0, 1, 2}, m = f 2^r in [0.5, 4);
//   2. y ~ m^(-1/3) by Newton's iteration for the inverse cube root,
//      y <- y + y (1 - m y^3) / 3, from a quadratic start (no division);
//   3. z = m y^2 ~ m^(1/3); the residual z^3 - m is evaluated with the
//      error-free products of fma (z^2 = p_h + p_l exactly, p_h z = t_h + t_l
//      exactly, t_h - m exact by Sterbenz's lemma), and one Newton step in
//      double-double gives cbrt(m) = z - res y^2 / 3 (y^2 = 1 / z^2 to working
//      precision);
//   4. ln(x), which enters the result scaled by 2^-54 / 3, as e' ln 2 +
//      2 atanh(s), s = (f' - 1) / (f' + 1), f' in [1/sqrt 2, sqrt 2), by its
//      odd series (absolute error below 1e-15);
//   5. the double-double value times (1 - 2^-54 ln(x)/3) is rounded once to
//      double and scaled by 2^q (exact).
// The result differs from the correctly rounded x^c only when x^c lies within
// about 2^-100 relative of a midpoint between two doubles.
//
// Most depths take a shorter way (pow_third_near): steps 2-5 on x itself from
// a single-precision start, with a rounding test that sends the values too
// near a midpoint for its accuracy to the full method.  Both give the
// correctly rounded value, so the device's and the host's single-precision
// functions may differ and the result does not: the strict kernels and the
// oracle (which evaluates the same expression as a correctly rounded pow)
// agree bit for bit.
#pragma once

#include <cmath>

#if defined(__CUDACC__)
#define DGSWEM_HD __host__ __device__ __forceinline__
#else
#define DGSWEM_HD inline
#endif

namespace dgswem {

// ln(x) = e' ln 2 + 2 atanh(s) for x = f 2^e, to 1e-15 absolute (step 4)
DGSWEM_HD double ln_series(double f, int e) {
  double fp = f;
  int ep = e;
  if (fp < 0.70710678118654752440) {
    fp = fp + fp;
    ep = ep - 1;
  }
  const double s = (fp - 1.0) / (fp + 1.0);
  const double s2 = s * s;
  double poly = 1.0 / 19.0;
  poly = 1.0 / 17.0 + s2 * poly;
  poly = 1.0 / 15.0 + s2 * poly;
  poly = 1.0 / 13.0 + s2 * poly;
  poly = 1.0 / 11.0 + s2 * poly;
  poly = 1.0 / 9.0 + s2 * poly;
  poly = 1.0 / 7.0 + s2 * poly;
  poly = 1.0 / 5.0 + s2 * poly;
  poly = 1.0 / 3.0 + s2 * poly;
  const double lnf = 2.0 * s + 2.0 * s * (s2 * poly);
  // ln 2 = hi + lo, hi with 21 trailing zero bits so that ep * hi is exact
  const double ln2_hi = 0x1.62e42feep-1;
  const double ln2_lo = 1.9082149292705877e-10;
  return (double)ep * ln2_hi + ((double)ep * ln2_lo + lnf);
}

// The method for every x (out of line: the kernels reach it once in 2^17
// calls, or outside the range of pow_third_near).
#if defined(__CUDACC__)
inline __host__ __device__ __noinline__
#else
inline
#endif
double pow_third_any(double x) {
  if (!(x > 0.0) || !(x < INFINITY)) {
    // pow(x, c) of a zero, negative, infinite or NaN base: 0, NaN, inf, NaN
    if (x == 0.0) return 0.0;
    if (x > 0.0) return x;
    return NAN;
  }
  int e;
  const double f = frexp(x, &e);  // x = f 2^e, f in [0.5, 1)
  // e = 3q + r, r in {0, 1, 2} (floor division for negative e)
  int q = e >= 0 ? e / 3 : -((-e + 2) / 3);
  const int r = e - 3 * q;
  const double m = ldexp(f, r);  // [0.5, 4)
  // step 2: inverse cube root, quadratic start (least-squares fit of the
  // relative error over [0.5, 4), below 9 %; five steps reach rounding level)
  double y = 1.31600226 + m * (-0.3495224 + m * 0.04591333);
  const double third = 1.0 / 3.0;
  for (int it = 0; it < 5; ++it) {
    const double y3 = y * y * y;
    y = y + y * ((1.0 - m * y3) * third);
  }
  // step 3: z ~ m^(1/3) and its double-double Newton correction
  const double y2 = y * y;
  const double z = m * y2;
  const double p_h = z * z;
  const double p_l = fma(z, z, -p_h);
  const double t_h = p_h * z;
  const double t_l = fma(p_h, z, -t_h);
  const double res = (t_h - m) + (t_l + p_l * z);
  const double corr = (res * y2) * third;  // cbrt(m) = z - corr
  const double k54 = 5.5511151231257827e-17 * third;  // 2^-54 / 3
  const double delta = ln_series(f, e) * k54;
  const double tail = (-corr - z * delta) + corr * delta;
  return ldexp(z + tail, q);
}

// Steps 2-5 for x in [2^-30, 2^30] (every depth of a run), without the
// scaling of step 1: started from l2 ~ log2(x), to 2^-17 absolute, and
// y0 ~ x^(-1/3), to 2^-19 relative.  One cubically convergent step takes u =
// x y0^2 to z ~ x^(1/3): with e = 1 - x y0^3 (below 2^-17), x^(1/3) =
// u (1 - e)^(-2/3) = u (1 + 2/3 e + 5/9 e^2 + O(e^3)).  The residual and the
// correction are those of step 3 (1 / z^2 as y0^2 (1 + 2/3 e), good to 2^-35,
// which the correction's own size, 2^-51, takes to 2^-86), and ln(x) = l2
// ln 2 is known to 2^-17.5, so z + tail has a relative error below 2^-72.
// Rounding both z + tail - 2^-71 z and z + tail + 2^-71 z (Ziv's test): equal
// values are the correctly rounded one (true); otherwise -- about once in
// 2^17 calls -- the result is left to pow_third_any (false).
DGSWEM_HD bool pow_third_near(double x, float l2, float y0f, double* out) {
  const double y0 = (double)y0f;
  const double u = x * y0 * y0;
  const double e = fma(-u, y0, 1.0);
  const double z = fma(u, e * fma(e, 5.0 / 9.0, 2.0 / 3.0), u);
  const double p_h = z * z;
  const double p_l = fma(z, z, -p_h);
  const double t_h = p_h * z;
  const double t_l = fma(p_h, z, -t_h);
  const double res = (t_h - x) + fma(p_l, z, t_l);
  const double w = (y0 * (1.0 / 3.0)) * y0;
  const double corr = res * fma(w, e * (2.0 / 3.0), w);
  const double delta = (double)(l2 * (0.69314718f * (5.5511151e-17f / 3.0f)));  // ln(x) 2^-54 / 3
  const double tail = fma(-z, delta, -corr);
  const double lo = z + fma(z, -0x1p-71, tail), hi = z + fma(z, 0x1p-71, tail);
  *out = hi;
  return lo == hi;
}

// pow_third_near with its start: the value, and whether it holds (x in range
// and the rounding test passed)
DGSWEM_HD bool pow_third_try(double x, double* out) {
#if defined(__CUDA_ARCH__)
  const float l2 = __log2f((float)x);
  float y0;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(l2 * (-1.0f / 3.0f)));
#else
  const float l2 = std::log2((float)x), y0 = std::exp2(l2 * (-1.0f / 3.0f));
#endif
  const bool near = pow_third_near(x, l2, y0, out);
  return near && x >= 0x1p-30 && x <= 0x1p30;
}

// DEPTH**(1.D0/3.D0), correctly rounded.  The start comes from the base-2
// single-precision logarithm and exponential (on the device the approximate
// instructions: lg2 within 2^-22 relative, so 30 * 2^-22 < 2^-17 here).
// 24 double-precision operations where pow_third_any's five Newton steps,
// frexp and ldexp take about 70 and three times as many integer ones: the
// strict stage kernel's volume terms take 2,200 cycles a tile of 128 elements
// now, 3,900 before.  kNear = false takes pow_third_any for every x (for tests).
template <bool kNear = true>
DGSWEM_HD double pow_third(double x) {
  double r;
  if (kNear && pow_third_try(x, &r)) return r;
  return pow_third_any(x);
}

// x / 3, correctly rounded, without a division: q = RN(x t), t = RN(1/3);
// r = x - 3q is exact (q is within 1 ulp of x/3, so r is a multiple of
// ulp(q) no larger than 3 ulp(q)) and fma(r, t, q) = RN(q + r t) is within
// 2^-53 ulp of x/3.  The exact quotient x/3 = M 2^e / 3 lies at least 1/6
// ulp from every midpoint between doubles (its remainder in ulps is a
// multiple of 1/3), so that rounding is the correctly rounded x/3 -- the IEEE
// division's result -- for every finite x.  The sign is x's (a zero quotient
// keeps the sign of x, as the division's does, which the sequence alone
// would lose: fma(+0, t, -0) = +0).  Four instructions instead of a division
// sequence.
DGSWEM_HD double div3(double x) {
  const double t = 1.0 / 3.0;
  const double q = x * t;
  const double r = fma(-q, 3.0, x);
  return copysign(fma(r, t, q), x);
}

// ---- reciprocal, quotient and square root, correctly rounded -----------------
// The IEEE results of 1 / x, a / b and sqrt(x) from a seed of about 20 bits, by
// one step of cubic convergence and Markstein's final step (P. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor",
// 1990: the residual of a result within an ulp is exact in one fma, and a
// second fma rounds the corrected result once).  For arguments in mid_range
// only, where no intermediate under- or overflows; the caller tests the range
// of all the values of a point at once and takes the operators for the rest,
// instead of a test and a branch in every operation.
//
// Reciprocal: y0 = (1 - e0) / x, |e0| <= 2^-19.9.  y1 = y0 + y0 (e0 + e0^2) =
// (1 - e0^3) / x up to one rounding: within 0.6 ulp.  e1 = 1 - x y1 is exact,
// and y1 + y1 e1 = (1 - e1^2) / x, |e1| < 2^-52, is rounded once: the correct
// rounding unless 1 / x lies above a midpoint by less than 2^-104 of itself,
// that is 2^106 - M X = k for a 53-bit X, an odd 54-bit M and k <= 4.
// Square root: with y0 ~ 1 / sqrt(a) to 2^-19.9, g0 = a y0, h0 = y0 / 2, r =
// 1/2 - g0 h0, both are multiplied by 1 + r + 3/2 r^2 ((1 - 2r)^(-1/2) up to
// 5/2 r^3); d = a - g1^2 is exact and g1 + d h1 lies within 2^-103 of sqrt(a),
// so its rounding is correct unless sqrt(a) is that near a midpoint, M^2 - 4 A
// = k (A the 53-bit mantissa times a power of two, M odd), |k| < 128.
// The few arguments so near a midpoint are all listed and tested, with every
// seed within the bounds, in tests/test_rounded_ops.py: only a significand of
// all ones can be rounded wrongly, in both, and mid_range leaves it out.
DGSWEM_HD double rcp_from(double x, double y0) {
  const double e0 = fma(-x, y0, 1.0);
  const double y1 = fma(y0, fma(e0, e0, e0), y0);
  return fma(fma(-x, y1, 1.0), y1, y1);
}
// a / b with y = 1 / b correctly rounded (Markstein): q is within an ulp
DGSWEM_HD double quot_from(double a, double b, double y) {
  const double q = a * y;
  return fma(fma(-b, q, a), y, q);
}
DGSWEM_HD double sqrt_from(double a, double y0) {
  const double g0 = a * y0, h0 = 0.5 * y0;
  const double r = fma(-g0, h0, 0.5);
  const double c = fma(1.5 * r, r, r);
  const double g1 = fma(g0, c, g0), h1 = fma(h0, c, h0);
  return fma(fma(-g1, g1, a), h1, g1);
}

#if defined(__CUDACC__)
// positive, between 2^-256 and 2^256 and not all ones in the significand's low
// word
__device__ __forceinline__ bool mid_range(double x) {
  return (unsigned)(__double2hiint(x) - 0x2ff00000) < 0x20000000u && __double2loint(x) != -1;
}
// seeds: the approximate instructions, which read the high 32 bits (relative
// errors over every high word of two binades, measured: 2^-19.9 and 2^-20.0)
__device__ __forceinline__ double rcp_seed(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ double rsqrt_seed(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
#endif

}  // namespace dgswem
