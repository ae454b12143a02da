// Double exp and log rounded to nearest, for the few transcendental terms of
// the evolution objective and of the PLS class coarsening, whose host
// counterparts (glibc exp / log) are correctly rounded in all but rare cases.
//
// Method (no vendor code): double-double arithmetic built from the
// error-free transformations of Knuth (TwoSum) and Dekker (TwoProduct via
// fma).
//   exp(x): Cody-Waite reduction x = k ln2 + r with ln 2 split into three
//           doubles, s = r / 2^10, expm1(s) by its Taylor series to degree 9
//           in Horner form, ten squarings through expm1(2t) = 2 e + e^2,
//           then 2^k (1 + e).  Relative error below 2^-92.
//   log(x): one Newton step on exp from a faithful start y0:
//           y = y0 + (x - e^y0) / e^y0, with e^y0 in double-double.
// The returned double is the nearest to the double-double value, so it is
// the correctly rounded result unless the exact value lies within ~2^-92
// (relative) of a rounding midpoint.
#pragma once

#include <math.h>

namespace kgb {

struct DD {
  double hi, lo;
};

__device__ __forceinline__ DD dd_two_sum(double a, double b) {
  const double s = __dadd_rn(a, b);
  const double bb = __dsub_rn(s, a);
  const double e = __dadd_rn(__dsub_rn(a, __dsub_rn(s, bb)), __dsub_rn(b, bb));
  return {s, e};
}

__device__ __forceinline__ DD dd_fast_two_sum(double a, double b) {
  const double s = __dadd_rn(a, b);
  return {s, __dsub_rn(b, __dsub_rn(s, a))};
}

__device__ __forceinline__ DD dd_two_prod(double a, double b) {
  const double p = __dmul_rn(a, b);
  return {p, fma(a, b, -p)};
}

__device__ __forceinline__ DD dd_add(DD a, DD b) {
  DD s = dd_two_sum(a.hi, b.hi);
  const DD t = dd_two_sum(a.lo, b.lo);
  s.lo = __dadd_rn(s.lo, t.hi);
  s = dd_fast_two_sum(s.hi, s.lo);
  s.lo = __dadd_rn(s.lo, t.lo);
  return dd_fast_two_sum(s.hi, s.lo);
}

__device__ __forceinline__ DD dd_mul(DD a, DD b) {
  DD p = dd_two_prod(a.hi, b.hi);
  p.lo = __dadd_rn(p.lo, __dadd_rn(__dmul_rn(a.hi, b.lo), __dmul_rn(a.lo, b.hi)));
  return dd_fast_two_sum(p.hi, p.lo);
}

__device__ __forceinline__ DD dd_div(DD a, DD b) {
  const double q1 = __ddiv_rn(a.hi, b.hi);
  DD t = dd_mul(b, DD{q1, 0.0});
  DD r = dd_add(a, DD{-t.hi, -t.lo});
  const double q2 = __ddiv_rn(r.hi, b.hi);
  t = dd_mul(b, DD{q2, 0.0});
  r = dd_add(r, DD{-t.hi, -t.lo});
  const double q3 = __ddiv_rn(r.hi, b.hi);
  DD q = dd_fast_two_sum(q1, q2);
  return dd_add(q, DD{q3, 0.0});
}

// e^x - 1 for |x| <= ln2/2 as a double-double.
__device__ inline DD dd_expm1_reduced(DD r) {
  const DD s{ldexp(r.hi, -10), ldexp(r.lo, -10)};
  // Horner: q = 1/9!; q = q s + 1/i! (i = 8..1); e = q s
  double fact = 362880.0;  // 9!
  DD q = dd_div(DD{1.0, 0.0}, DD{fact, 0.0});
  for (int i = 8; i >= 1; --i) {
    fact /= static_cast<double>(i + 1);  // i! (exact)
    q = dd_add(dd_mul(q, s), dd_div(DD{1.0, 0.0}, DD{fact, 0.0}));
  }
  DD e = dd_mul(q, s);
  for (int k = 0; k < 10; ++k) e = dd_add(DD{2.0 * e.hi, 2.0 * e.lo}, dd_mul(e, e));
  return e;
}

// e^x as a double-double mantissa and a power of two: e^x = (1 + e) 2^k.
__device__ inline DD dd_exp_parts(double x, int& k_out) {
  const double kLn2a = 0x1.62e42fefa39efp-1, kLn2b = 0x1.abc9e3b39803fp-56, kLn2c = 0x1.7b57a079a1934p-111;
  const double kInvLn2 = 0x1.71547652b82fep+0;
  const double k = rint(__dmul_rn(x, kInvLn2));
  DD p = dd_two_prod(k, kLn2a);
  DD r = dd_add(DD{x, 0.0}, DD{-p.hi, -p.lo});
  p = dd_two_prod(k, kLn2b);
  r = dd_add(r, DD{-p.hi, -p.lo});
  r = dd_add(r, DD{-__dmul_rn(k, kLn2c), 0.0});
  k_out = static_cast<int>(k);
  return dd_expm1_reduced(r);
}

// The quick path: x = (32 k + j) ln2 / 32 + r, |r| <= ln2 / 64, and
// e^r - 1 = r + r^2 / 2 + t with r and r^2 / 2 in two doubles and the tail t, below
// 2^-21, in one.  Products and sums of the low parts are within 2^-74 of
// e^r - 1 <= 2^-6, the series ends before r^9 / 9! < 2^-77, and the table is good to
// 2^-106: together below 2^-66 of the result, which is tested for a rounding
// midpoint within that distance (one call in about 8000 goes on to the series
// above).  About 60 dependent FP64 operations of 64 cycles each; the series with
// its nine double-double divisions is some 1500.
struct ExpParts {
  DD one;    // (1 + e) = e^x 2^-k
  DD e;      // e^r - 1
  int k, j;
};

__device__ inline ExpParts exp_parts_quick(double x) {
  // 2^(j / 32) in two doubles
  static const double kPow[32][2] = {
    {0x1.0000000000000p+0, 0x0.0p+0}, {0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55},
    {0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54}, {0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54},
    {0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55}, {0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54},
    {0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54}, {0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55},
    {0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55}, {0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54},
    {0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55}, {0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59},
    {0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56}, {0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55},
    {0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54}, {0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54},
    {0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54}, {0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55},
    {0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55}, {0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54},
    {0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54}, {0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57},
    {0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56}, {0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54},
    {0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54}, {0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56},
    {0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55}, {0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56},
    {0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55}, {0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54},
    {0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54}, {0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54},
  };
  const double kLn2a = 0x1.62e42fefa39efp-6, kLn2b = 0x1.abc9e3b39803fp-61;  // ln 2 / 32
  const double k32Ln2 = 0x1.71547652b82fep+5;                                // 32 / ln 2
  const double n = rint(__dmul_rn(x, k32Ln2));
  const int ni = static_cast<int>(n);
  ExpParts out;
  out.j = ni & 31;
  out.k = (ni - out.j) / 32;
  const DD p = dd_two_prod(n, kLn2a);
  const DD d = dd_two_sum(x, -p.hi);
  const DD r = dd_fast_two_sum(d.hi, __dsub_rn(__dsub_rn(d.lo, p.lo), __dmul_rn(n, kLn2b)));
  const DD q = dd_two_prod(r.hi, r.hi);
  const double h = 0.5 * q.hi, l = fma(r.hi, r.lo, 0.5 * q.lo);
  double t = fma(r.hi, 1.0 / 40320.0, 1.0 / 5040.0);
  t = fma(r.hi, t, 1.0 / 720.0);
  t = fma(r.hi, t, 1.0 / 120.0);
  t = fma(r.hi, t, 1.0 / 24.0);
  t = fma(r.hi, t, 1.0 / 6.0);
  t = __dmul_rn(__dmul_rn(q.hi, r.hi), t);
  const DD s = dd_fast_two_sum(r.hi, h);
  out.e = dd_fast_two_sum(s.hi, __dadd_rn(t, __dadd_rn(__dadd_rn(r.lo, l), s.lo)));
  const double th = kPow[out.j][0], tl = kPow[out.j][1];
  const DD m = dd_two_prod(th, out.e.hi);
  const DD u = dd_fast_two_sum(th, m.hi);
  const double lo = __dadd_rn(__dadd_rn(u.lo, fma(tl, out.e.hi, m.lo)), fma(th, out.e.lo, tl));
  out.one = dd_fast_two_sum(u.hi, lo);
  return out;
}

// hi + lo where every value within err of it rounds to the same double, else NaN.
__device__ __forceinline__ double rounded_or_nan(double hi, double lo, double err) {
  const double a = __dadd_rn(hi, __dsub_rn(lo, err)), b = __dadd_rn(hi, __dadd_rn(lo, err));
  return a == b ? a : NAN;
}

__device__ __noinline__ double cr_exp_series(double x) {
  int k = 0;
  const DD e = dd_exp_parts(x, k);
  const DD m = dd_add(DD{1.0, 0.0}, e);
  // 2^k (hi + lo): scale both parts in two steps so no intermediate overflows
  const int k1 = k / 2, k2 = k - k1;
  return ldexp(ldexp(__dadd_rn(m.hi, m.lo), k1), k2);
}

__device__ inline double cr_exp(double x) {
  if (isnan(x)) return x;
  if (x > 709.79) return INFINITY;
  if (x < -745.2) return 0.0;
  const ExpParts p = exp_parts_quick(x);
  const double v = rounded_or_nan(p.one.hi, p.one.lo, 0x1p-65);
  if (isnan(v)) return cr_exp_series(x);
  const int k1 = p.k / 2, k2 = p.k - k1;
  return ldexp(ldexp(v, k1), k2);
}

__device__ __noinline__ double cr_log_series(double x, double y0) {
  int k = 0;
  const DD e = dd_exp_parts(y0, k);
  // E = e^y0 = (1 + e) 2^k; d = (x - E) / E
  const DD one_e = dd_add(DD{1.0, 0.0}, e);
  const DD E{ldexp(one_e.hi, k), ldexp(one_e.lo, k)};
  const DD num = dd_add(DD{x, 0.0}, DD{-E.hi, -E.lo});
  const double d = __ddiv_rn(num.hi, E.hi);
  return __dadd_rn(y0, d);
}

__device__ inline double cr_log(double x) {
  if (isnan(x) || x < 0.0) return NAN;
  if (x == 0.0) return -INFINITY;
  if (isinf(x)) return INFINITY;
  if (x == 1.0) return 0.0;
  const double y0 = log(x);
  const ExpParts p = exp_parts_quick(y0);
  // d = (x - e^y0) / e^y0: near x = 1 against e^y0 - 1 itself, whose error is a
  // part of y0; else against e^y0 2^-k
  const bool near = p.k == 0 && p.j == 0;
  double num;
  if (near) num = __dsub_rn(__dsub_rn(__dsub_rn(x, 1.0), p.e.hi), p.e.lo);
  else num = __dsub_rn(__dsub_rn(ldexp(x, -p.k), p.one.hi), p.one.lo);
  const double v = rounded_or_nan(y0, __ddiv_rn(num, p.one.hi), near ? fabs(y0) * 0x1p-65 : 0x1p-65);
  return isnan(v) ? cr_log_series(x, y0) : v;
}

}  // namespace kgb
