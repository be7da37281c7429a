// Correctly rounded exp(x), log(x), x^y and x^(1/4) in FP64, for the
// transport coefficients (zeta/s forms 1-5, src/trancoeff.cpp:19-70),
// EoSChiral's power law, EoSHadron's logarithmic table coordinates and the
// entropy-to-energy inversion of the initial states (src/s95p.cpp:14-40).  The reference
// evaluates them with the host C library, whose exp and pow are accurate to
// about half an ulp; returning the correctly rounded value reproduces the
// library's result except where the exact value lies within ~1e-3 ulp of a
// rounding boundary, while a faithfully rounded device exp (up to 1 ulp)
// differs from it in a sizeable fraction of calls.  Bulk viscosity amplifies
// a last-bit difference by ~1e6 within ten steps near the limiter and the
// vacuum edge, so the last bit matters for parity.
//
// Method (own implementation from the mathematics, double-double arithmetic
// after Dekker (1971) and Knuth's two-sum; constants from
// gen_crmath_consts.py, exact rational arithmetic):
//   exp: k = rint(x / ln 2); r = x - k ln 2 with ln 2 split into three
//        doubles (Cody & Waite 1980); s = r / 2^8; expm1(s) by its Taylor
//        series to s^11 / 11! in double-double (|s| < 1.4e-3, truncation
//        < 2^-125); eight doublings expm1(2a) = 2 expm1(a) + expm1(a)^2;
//        1 + expm1 rounded to nearest once; scaled by 2^k, with the
//        subnormal range rounded to integer multiples of 2^-1074 from the
//        double-double.  Relative error before the final rounding < 2^-98.
//   log: a Newton step on the exp above from a faithful seed (log_cr).
//   x^y: exp of y log(x), both in double-double (pow_cr).
//   exp and x^y first take a short form (exp_try, log_short; Ziv's strategy,
//        ACM TOMS 17 (1991)): tables of 2^(j/64) and of log at 1/128 steps
//        (Tang's table method, ACM TOMS 15 (1989) and 16 (1990), the first
//        two orders of each series in double-double), whose result is taken
//        when its error bound cannot move the rounding; the forms above
//        decide the rest, about one argument in eight thousand.
//   x^(1/4): sqrt(x) as a double-double (the correctly rounded square root
//        and its exact residual by fma), its square root the same way, and
//        one rounding of the sum.
// Every operation is an IEEE add, multiply, divide, sqrt or an explicit fma,
// none contracted (the library builds with -fmad=false), so host and device
// compilations of this header give the same bits.
#pragma once

#include <math.h>

#include "vh_crmath_tab.cuh"

#ifdef __CUDACC__
#define VH_CRM __host__ __device__ __forceinline__
// the long forms stay out of line: they run for one argument in thousands
#define VH_CRM_COLD static __host__ __device__ __noinline__
#else
#define VH_CRM static inline
#define VH_CRM_COLD static inline
#endif

namespace vh {
namespace crm {

struct dd {
  double hi, lo;
};

#ifdef __CUDACC__
static __device__ const double kExpTabDev[128] = {VH_CRM_EXP_TAB};
static __device__ const double kLogTabDev[384] = {VH_CRM_LOG_TAB};
#endif
static const double kExpTabHost[128] = {VH_CRM_EXP_TAB};
static const double kLogTabHost[384] = {VH_CRM_LOG_TAB};
VH_CRM double exp_tab(int k) {
#ifdef __CUDA_ARCH__
  return __ldg(kExpTabDev + k);
#else
  return kExpTabHost[k];
#endif
}
VH_CRM double log_tab(int k) {
#ifdef __CUDA_ARCH__
  return __ldg(kLogTabDev + k);
#else
  return kLogTabHost[k];
#endif
}

VH_CRM dd two_sum(double a, double b) {
  const double s = a + b;
  const double bb = s - a;
  const double e = (a - (s - bb)) + (b - bb);
  return {s, e};
}

VH_CRM dd fast_two_sum(double a, double b) {  // |a| >= |b|
  const double s = a + b;
  return {s, b - (s - a)};
}

VH_CRM dd two_prod(double a, double b) {
  const double p = a * b;
  return {p, fma(a, b, -p)};
}

VH_CRM dd add(dd a, dd b) {
  dd s = two_sum(a.hi, b.hi);
  const dd t = two_sum(a.lo, b.lo);
  s.lo += t.hi;
  s = fast_two_sum(s.hi, s.lo);
  s.lo += t.lo;
  return fast_two_sum(s.hi, s.lo);
}

VH_CRM dd mul(dd a, dd b) {
  dd p = two_prod(a.hi, b.hi);
  const double c = a.hi * b.lo;
  const double d = a.lo * b.hi;
  p.lo += c + d;
  return fast_two_sum(p.hi, p.lo);
}

// 2^k for -1022 <= k <= 1023, built from its bit pattern
VH_CRM double pow2i(int k) {
  const long long bits = (long long)(k + 1023) << 52;
#ifdef __CUDA_ARCH__
  return __longlong_as_double(bits);
#else
  double d;
  __builtin_memcpy(&d, &bits, sizeof d);
  return d;
#endif
}

// y * 2^k rounded once, y = hi + lo in [0.7, 1.5), |k| <= 1100
VH_CRM double scale_round(dd y, int k) {
  if (k > 1023) return y.hi * pow2i(1023) * pow2i(k - 1023);  // may overflow to inf
  if (k > -1022) return y.hi * pow2i(k);                        // exact
  // subnormal range: count units of 2^-1074
  const int sh = k + 1074;
  if (sh < -1) return 0.0;  // y 2^k < 2^-1075.4, below half the smallest subnormal
  const double f = sh >= 0 ? pow2i(sh) : 0.5;
  const double zh = y.hi * f, zl = y.lo * f;  // exact
  double n = rint(zh);
  const double rem = (zh - n) + zl;
  if (rem > 0.5) {
    n += 1.0;
  } else if (rem < -0.5) {
    n -= 1.0;
  } else if (rem == 0.5 || rem == -0.5) {  // tie: to even
    const double m = n + (rem > 0 ? 1.0 : -1.0);
    if (fmod(m, 2.0) == 0.0) n = m;
  }
  return n * pow2i(-1022) * pow2i(-52);  // exact: n < 2^53
}

// ln 2 = LN2_1 + LN2_2 + LN2_3 (LN2_1 has 33 significant bits, so k LN2_1
// is exact for |k| < 2^20)
#define VH_CRM_LN2_1 0x1.62e42fef00000p-1
#define VH_CRM_LN2_2 0x1.473de6af278edp-34
#define VH_CRM_LN2_3 -0x1.9ff0342542fc3p-90

// expm1(r) for |r| <= 0.36 as a double-double
VH_CRM dd expm1_dd(dd r) {
  // s = r / 2^8
  const dd s = {r.hi * 0x1p-8, r.lo * 0x1p-8};
  // expm1(s) = s (1 + s/2! + s^2/3! + ... + s^10/11!) by Horner
  const dd c[12] = {{0., 0.},
                    {0x1.0000000000000p+0, 0.},
                    {0x1.0000000000000p-1, 0.},
                    {0x1.5555555555555p-3, 0x1.5555555555555p-57},
                    {0x1.5555555555555p-5, 0x1.5555555555555p-59},
                    {0x1.1111111111111p-7, 0x1.1111111111111p-63},
                    {0x1.6c16c16c16c17p-10, -0x1.f49f49f49f49fp-65},
                    {0x1.a01a01a01a01ap-13, 0x1.a01a01a01a01ap-73},
                    {0x1.a01a01a01a01ap-16, 0x1.a01a01a01a01ap-76},
                    {0x1.71de3a556c734p-19, -0x1.c154f8ddc6c00p-73},
                    {0x1.27e4fb7789f5cp-22, 0x1.cbbc05b4fa99ap-76},
                    {0x1.ae64567f544e4p-26, -0x1.c062e06d1f209p-80}};
  dd p = c[11];
#pragma unroll
  for (int n = 10; n >= 1; n--) p = add(mul(p, s), c[n]);
  dd e = mul(p, s);
  // expm1(2a) = 2 expm1(a) + expm1(a)^2, eight times
#pragma unroll
  for (int j = 0; j < 8; j++) e = add({2. * e.hi, 2. * e.lo}, mul(e, e));
  return e;
}

VH_CRM_COLD double exp_long(double x) {
  if (!(x == x)) return x;  // NaN
  if (x > 709.8) return (double)INFINITY;
  if (x < -746.0) return 0.0;
  const double INV_LN2 = 0x1.71547652b82fep+0;
  const double k = rint(x * INV_LN2);
  // r = x - k ln2 as a double-double
  dd r = two_sum(x, -(k * VH_CRM_LN2_1));  // k * LN2_1 exact
  r = add(r, {-two_prod(k, VH_CRM_LN2_2).hi, -two_prod(k, VH_CRM_LN2_2).lo});
  r = add(r, {-(k * VH_CRM_LN2_3), 0.0});
  const dd y = add({1.0, 0.0}, expm1_dd(r));
  return scale_round(y, (int)k);
}

VH_CRM double from_bits(unsigned long long u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double d;
  __builtin_memcpy(&d, &u, sizeof d);
  return d;
#endif
}

VH_CRM unsigned long long to_bits(double d) {
#ifdef __CUDA_ARCH__
  return (unsigned long long)__double_as_longlong(d);
#else
  unsigned long long u;
  __builtin_memcpy(&u, &d, sizeof u);
  return u;
#endif
}

// log(x), correctly rounded.  x = m 2^k with m in [0.707, 1.415); the
// platform's log(m) (faithful, on the host or the device) is a seed y0;
// one Newton step on exp, y = y0 + ((m - 1) - expm1(y0)) / exp(y0), with
// m - 1 exact and expm1(y0) a double-double, removes the seed's error (the
// step's own error is of the order of the seed error squared, ~2^-104 |y|);
// then k ln 2 + y in double-double and one rounding.  Seeds that differ by
// an ulp give the same result, so host and device agree.
VH_CRM dd log_dd(double x);

VH_CRM double log_cr(double x) {
  if (!(x > 0.)) return x == 0. ? -(double)INFINITY : (double)NAN;
  if (x == (double)INFINITY) return x;
  return log_dd(x).hi;
}

// log(x) as a double-double for finite x > 0 (relative error ~2^-102):
// the steps of log_cr before its one rounding
VH_CRM dd log_dd(double x) {
  int k = 0;
  if (x < 0x1p-1022) {  // subnormal: scale into the normal range (exact)
    x *= 0x1p54;
    k = -54;
  }
  const unsigned long long u = to_bits(x);
  k += (int)(u >> 52) - 1023;
  double m = from_bits((u & 0x000fffffffffffffull) | 0x3ff0000000000000ull);  // [1, 2)
  if (m > 1.41421356) {
    m *= 0.5;
    k += 1;
  }
  const double y0 = log(m);
  const dd em1 = expm1_dd({y0, 0.});
  const dd d = add({m - 1., 0.}, {-em1.hi, -em1.lo});  // m - 1 exact (Sterbenz)
  const double c = d.hi / (1. + em1.hi);
  const dd y = two_sum(y0, c);
  const double kd = (double)k;
  dd L = add(two_prod(kd, VH_CRM_LN2_2), {kd * VH_CRM_LN2_3, 0.});
  L = add({kd * VH_CRM_LN2_1, 0.}, L);
  return add(L, y);
}

// exp(t.hi + t.lo) for a double-double argument (|t.lo| <= ulp(t.hi)), as
// exp_cr: the low part joins the reduced argument before expm1
VH_CRM double exp_dd_cr(dd t) {
  const double x = t.hi;
  if (!(x == x)) return x;  // NaN
  if (x > 709.8) return (double)INFINITY;
  if (x < -746.0) return 0.0;
  const double INV_LN2 = 0x1.71547652b82fep+0;
  const double k = rint(x * INV_LN2);
  dd r = two_sum(x, -(k * VH_CRM_LN2_1));
  r = add(r, {-two_prod(k, VH_CRM_LN2_2).hi, -two_prod(k, VH_CRM_LN2_2).lo});
  r = add(r, {-(k * VH_CRM_LN2_3), t.lo});
  const dd y = add({1.0, 0.0}, expm1_dd(r));
  return scale_round(y, (int)k);
}

// x^y, correctly rounded but where the exact value lies within ~2^-38 ulp
// of a rounding boundary: exp(y log x) with log x a double-double
// (log_dd), the product y log x a double-double (absolute error below
// 2^-92 while it is in exp's range) and exp_dd_cr.  y = 2 is x * x (one
// rounding of the exact square, which can be a tie).  The C library's
// special values: x^0 = 1 and 1^y = 1 (NaN included), NaN otherwise
// propagates; 0^y = +0 (y > 0) or +inf (y < 0), with -0 kept for odd
// integers y; inf^y = inf or 0; negative x for integer y only (NaN else).
VH_CRM_COLD double pow_long(double x, double y) {
  if (y == 0. || x == 1.) return 1.;
  if (!(x == x) || !(y == y)) return x + y;
  if (y == 2.) return x * x;
  const bool yint = rint(y) == y;
  const bool yodd = yint && fabs(y) < 0x1p53 && fmod(y, 2.0) != 0.;
  if (x == 0.) {
    const double r = y > 0. ? 0. : (double)INFINITY;
    return (yodd && to_bits(x) >> 63) ? -r : r;
  }
  double sgn = 1.;
  if (x < 0.) {
    if (!yint) return (double)NAN;
    if (yodd) sgn = -1.;
    x = -x;
  }
  if (x == (double)INFINITY) return sgn * (y > 0. ? (double)INFINITY : 0.);
  const dd L = log_dd(x);
  const dd t = mul({y, 0.}, L);
  if (t.hi > 709.8) return sgn * (double)INFINITY;
  if (t.hi < -746.0) return sgn * 0.;
  return sgn * exp_dd_cr(t);
}

// exp(t.hi + t.lo) for |t.hi| <= 700, |t.lo| <= 2^-30, in the short form:
// t = k ln2/64 + r, |r| < 2^-7.5, 2^(j/64) (1 + r + r^2/2 + r^3 P(r)); true
// and the result in *out if the result's relative error, below 2^-72 plus
// t's own absolute error (at most 2^-70), leaves one double to round to.
VH_CRM bool exp_try(dd t, double* out) {
  const double k = rint(t.hi * VH_CRM_64_LN2);
  const double rh = fma(-k, VH_CRM_LN2_64H, t.hi);  // exact: k H has 53 bits
  const dd r = fast_two_sum(rh, fma(-k, VH_CRM_LN2_64L, t.lo));
  const dd r2 = two_prod(r.hi, r.hi);
  double P = 0x1.a01a01a01a01ap-16;  // 1/8!
  P = fma(P, r.hi, 0x1.a01a01a01a01ap-13);
  P = fma(P, r.hi, 0x1.6c16c16c16c17p-10);
  P = fma(P, r.hi, 0x1.1111111111111p-7);
  P = fma(P, r.hi, 0x1.5555555555555p-5);
  P = fma(P, r.hi, 0x1.5555555555555p-3);
  // q = exp(r) - 1
  const dd s = fast_two_sum(r.hi, 0.5 * r2.hi);
  const double ql = (r.hi * r2.hi) * P + (s.lo + (r.lo + (0.5 * r2.lo + r.hi * r.lo)));
  const dd q = fast_two_sum(s.hi, ql);
  const int n = (int)k, j = n & 63;
  const double th = exp_tab(2 * j), tl = exp_tab(2 * j + 1);
  const dd p = two_prod(th, q.hi);
  const dd a = fast_two_sum(th, p.hi);
  const dd y = fast_two_sum(a.hi, a.lo + (p.lo + (tl + (th * q.lo + tl * q.hi))));
  const double err = 0x1p-67 * y.hi;
  const double up = y.hi + (y.lo + err), down = y.hi + (y.lo - err);
  *out = up * pow2i((n - j) >> 6);  // exact: |t.hi| <= 700
  return up == down;
}

// log(x) for a normal x > 0 as a double-double, absolute error below 2^-73:
// x = 2^k m, m c = 1 + r with c the table's reciprocal near 1/m, |r| < 2^-7.9,
// k ln2 - log c + r - r^2/2 + r^3 P(r)
VH_CRM dd log_short(double x) {
  const unsigned long long u = to_bits(x);
  const double k = (double)((int)(u >> 52) - 1023);
  const double m = from_bits((u & 0x000fffffffffffffull) | 0x3ff0000000000000ull);
  const int i = 3 * (int)((u >> 45) & 127);
  const double c = log_tab(i);
  const dd mc = two_prod(m, c);
  const dd r = fast_two_sum(mc.hi - 1., mc.lo);
  const dd r2 = two_prod(r.hi, r.hi);
  double P = 0x1.c71c71c71c71cp-4;  // 1/9
  P = fma(P, r.hi, -0x1p-3);
  P = fma(P, r.hi, 0x1.2492492492492p-3);
  P = fma(P, r.hi, -0x1.5555555555555p-3);
  P = fma(P, r.hi, 0x1.999999999999ap-3);
  P = fma(P, r.hi, -0x1p-2);
  P = fma(P, r.hi, 0x1.5555555555555p-2);
  const dd s1 = two_sum(k * VH_CRM_LN2H, log_tab(i + 1));  // k H exact
  const dd s2 = two_sum(s1.hi, r.hi);
  const dd s3 = two_sum(s2.hi, -0.5 * r2.hi);
  const double lo = (r.hi * r2.hi) * P + (s3.lo + (s2.lo + (s1.lo + (r.lo - (0.5 * r2.lo + r.hi * r.lo) +
                    fma(k, VH_CRM_LN2L, log_tab(i + 2))))));
  return two_sum(s3.hi, lo);
}

VH_CRM double exp_cr(double x) {
  double r;
  if (fabs(x) <= 700. && exp_try({x, 0.}, &r)) return r;
  return exp_long(x);
}

// x^y for y not 0 or 2, |y| <= 8, with L = pow_base(x): the log of x once
// for all its powers (NaN where the short form does not apply)
VH_CRM dd pow_base(double x) {
  if (x >= 0x1p-1022 && x <= 0x1.fffffffffffffp1023 && x != 1.) return log_short(x);
  return {(double)NAN, 0.};
}
VH_CRM double pow_of(double x, dd L, double y) {
  const dd p = two_prod(y, L.hi);
  const dd t = fast_two_sum(p.hi, fma(y, L.lo, p.lo));
  double r;
  if (fabs(t.hi) <= 700. && exp_try(t, &r)) return r;
  return pow_long(x, y);
}
VH_CRM double pow_cr(double x, double y) {
  if (fabs(y) <= 8. && y != 2. && y != 0.) return pow_of(x, pow_base(x), y);
  return pow_long(x, y);
}

// x^(1/4) for x >= 0 (x = +0 gives +0, x = inf gives inf)
VH_CRM double root4_cr(double x) {
  if (!(x > 0.) || x == (double)INFINITY) return x < 0. ? (double)NAN : x;
  // a + al = sqrt(x): a correctly rounded, fma(-a, a, x) exact
  const double a = sqrt(x);
  const double al = fma(-a, a, x) / (2. * a);
  // b + bl = sqrt(a + al)
  const double b = sqrt(a);
  const double bl = (fma(-b, b, a) + al) / (2. * b);
  return b + bl;
}

// y / b correctly rounded, from r = RN(1/b), without a divide: the
// quotient q0 = RN(y r) is faithful, the remainder y - b q0 is exact in an
// fma, and RN(q0 + r (y - b q0)) = RN(y / b) (Markstein's theorem, IBM J.
// Res. Dev. 34 (1990); Muller et al., Handbook of Floating-Point
// Arithmetic, the Newton-Raphson division chapter).  It needs nothing to
// underflow or overflow: mk_num_ok(y) (2^-900 <= |y| < 2^900, or y = +-0)
// and mk_den_ok(b) (2^-100 <= b <= 2^100, so b > 0).  Callers test a batch
// of numerators once and divide the IEEE way otherwise, so that a batch of
// quotients is free of branches (a divide is an instruction sequence with a
// branch to a slow path, which keeps independent divides from overlapping).
// Both tests and the sign fix below are bit operations, off the FP64 pipe.
VH_CRM unsigned mk_hi(double y) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2hiint(y);
#else
  unsigned long long u;
  __builtin_memcpy(&u, &y, sizeof u);
  return (unsigned)(u >> 32);
#endif
}
VH_CRM unsigned mk_lo(double y) {
#ifdef __CUDA_ARCH__
  return (unsigned)__double2loint(y);
#else
  unsigned long long u;
  __builtin_memcpy(&u, &y, sizeof u);
  return (unsigned)u;
#endif
}
// |y| in [2^-900, 2^900): biased exponent in [123, 1922]; or y = +-0
VH_CRM bool mk_num_ok(double y) {
  const unsigned h = mk_hi(y) & 0x7fffffffu;
  return h - (123u << 20) < (1800u << 20) || (h | mk_lo(y)) == 0u;
}
VH_CRM bool mk_den_ok(double b) { return b >= 0x1p-100 && b <= 0x1p100; }
// For y != 0 the quotient has the sign of q0; for y = +-0 (b > 0) the
// divide returns y, which q0 = y r also is, so the sign of q0 is the sign
// of the result in both cases.
VH_CRM double mk_div(double y, double b, double r) {
  const double q0 = y * r;
  const double rem = fma(-q0, b, y);
  return copysign(fma(rem, r, q0), q0);
}

}  // namespace crm
}  // namespace vh

#undef VH_CRM
#undef VH_CRM_COLD
#undef VH_CRM_LN2_1
#undef VH_CRM_LN2_2
#undef VH_CRM_LN2_3
