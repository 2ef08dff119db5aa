// Double-float ("df64") arithmetic on the FP32 pipe: a value is an
// unevaluated sum hi + lo of two floats (about 48 significant bits).
//
// GB300 runs FP32 FMA ~60x faster than FP64 FMA (73 vs 1.2 TFLOP/s measured),
// so the FP64-accuracy products of the eigenpair refinement are evaluated in
// this arithmetic: error-free transformations TwoSum (Knuth, TAOCP vol. 2,
// 4.2.2) and TwoProduct via FMA, with the accurate (renormalising) addition
// of the double-double literature (e.g. Hida, Li, Bailey, "Algorithms for
// quad-double precision floating point arithmetic", ARITH 2001, restricted
// to two components). Relative error per operation is below ~2^-47.
#pragma once
#include "gla_common.cuh"

namespace gla {

struct df64 {
  float hi, lo;
};

GLA_DEV df64 df_make(float h, float l) {
  df64 r;
  r.hi = h;
  r.lo = l;
  return r;
}

// Exact: a + b = s + e.
GLA_DEV void two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// Exact when |a| >= |b| (or a == 0): a + b = s + e.
GLA_DEV void quick_two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  e = b - (s - a);
}

GLA_DEV df64 df_add(df64 a, df64 b) {
  float s, e;
  two_sum(a.hi, b.hi, s, e);
  e += a.lo + b.lo;
  df64 r;
  quick_two_sum(s, e, r.hi, r.lo);
  return r;
}

GLA_DEV df64 df_neg(df64 a) { return df_make(-a.hi, -a.lo); }

// acc + a * b (a, b double-float).
GLA_DEV df64 df_mac(df64 acc, df64 a, df64 b) {
  const float p = a.hi * b.hi;
  float pe = fmaf(a.hi, b.hi, -p);
  pe = fmaf(a.hi, b.lo, pe);
  pe = fmaf(a.lo, b.hi, pe);
  float s, e;
  two_sum(acc.hi, p, s, e);
  e += pe + acc.lo;
  df64 r;
  quick_two_sum(s, e, r.hi, r.lo);
  return r;
}

// acc + a * b (b a plain float).
GLA_DEV df64 df_mac(df64 acc, df64 a, float b) {
  const float p = a.hi * b;
  float pe = fmaf(a.hi, b, -p);
  pe = fmaf(a.lo, b, pe);
  float s, e;
  two_sum(acc.hi, p, s, e);
  e += pe + acc.lo;
  df64 r;
  quick_two_sum(s, e, r.hi, r.lo);
  return r;
}

GLA_DEV df64 df_mul(df64 a, df64 b) { return df_mac(df_make(0.f, 0.f), a, b); }

// A double as three floats (all 53 bits), and the difference of two rounded to
// a float: on the FP32 pipe and with no more error than a few of its roundings,
// however close the two are (the differences of the first and of the second
// parts are exact in two floats each, and what cancels, cancels exactly).
struct f3 {
  float hi, mid, lo;
};
GLA_DEV f3 f3_from(double x) {
  f3 r;
  r.hi = (float)x;
  x -= (double)r.hi;
  r.mid = (float)x;
  r.lo = (float)(x - (double)r.mid);
  return r;
}
GLA_DEV float f3_diff(f3 a, f3 b) {
  float s, e, t, f;
  two_sum(a.hi, -b.hi, s, e);
  two_sum(a.mid, -b.mid, t, f);
  return (s + t) + (e + (f + (a.lo - b.lo)));
}

// Conversions (FP64 instructions: use outside inner loops only).
GLA_DEV df64 df_from(double x) {
  const float h = (float)x;
  return df_make(h, (float)(x - (double)h));
}
// df_from(a 2^-se) for |a| 2^-se <= 1 on the integer pipe (df_from and ldexp
// take five FP64-pipe instructions, 64 cycles each for a warp, and ldexp's
// code is long where it is unrolled).
GLA_DEV df64 df_scaled(double a, int se) {
  unsigned long long b = (unsigned long long)__double_as_longlong(a);
  int e = (int)(b >> 52) & 0x7ff;
  if (e == 0) {  // zero or subnormal
    if (a == 0.0) return df_make(0.f, 0.f);
    b = (unsigned long long)__double_as_longlong(a * 0x1p54);
    e = ((int)(b >> 52) & 0x7ff) - 54;
  }
  const unsigned long long m = b & 0xfffffffffffffull;
  // biased exponent of hi as a float; small ones are built 2^128 larger
  const int ef = e - 1023 - se + 127, eb = min(ef < 64 ? ef + 128 : ef, 250);
  if (eb < 64) return df_make(0.f, 0.f);  // below 2^-190
  const unsigned sign = (unsigned)(b >> 32) & 0x80000000u;
  // hi: to nearest, ties to even, at bit 29 (a carry runs into the exponent)
  const unsigned ht = (unsigned)(m >> 29), hm = (unsigned)((m + 0xfffffffull + (ht & 1u)) >> 29);
  const int li = (int)((unsigned)m & 0x1fffffffu) - (int)((hm - ht) << 29);
  float hi = __uint_as_float(sign | (((unsigned)eb << 23) + hm));
  float lo = __uint_as_float(__float_as_uint((float)li * __int_as_float((eb - 52) << 23)) ^ sign);
  if (ef < 64) {
    hi = hi * 0x1p-64f * 0x1p-64f;
    lo = lo * 0x1p-64f * 0x1p-64f;
  }
  return df_make(hi, lo);
}
// df_from without the FP64 pipe for 2^-60 < |x| < 2^120.
GLA_DEV df64 df_from_fast(double x) {
  const int e = (int)((unsigned long long)__double_as_longlong(x) >> 52) & 0x7ff;
  return e > 1023 - 60 && e < 1023 + 120 ? df_scaled(x, 0) : df_from(x);
}
GLA_DEV double df_to(df64 a) { return (double)a.hi + (double)a.lo; }

}  // namespace gla
