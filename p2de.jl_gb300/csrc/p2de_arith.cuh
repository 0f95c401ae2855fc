// FP64 point arithmetic of the kernels: reciprocal, quotient, square root and logarithm with
// most of their work on the FP32 and integer pipes.
#pragma once

#include <cuda_runtime.h>

#include "p2de_tables.h"

namespace p2de {

// 1/x and sqrt(x) with most of the work off the FP64 pipe, which issues one warp instruction
// per 17-20 clocks and SM here: an FP32 approximation (2^-23) is refined to about 44 bits in
// FP32 and integer arithmetic (24-30 instructions on pipes that otherwise issue in a tenth of
// their slots), and one FP64 Newton-Raphson step y + y (1 - x y), or for the root the step
// g + (x - g g) y/2 from g = x y, y ~ 1/sqrt(x), gives the correctly rounded result unless it
// lies within about 2^-88 relative of a rounding tie. 2 and 3 FP64 operations, 36 and 52 SM
// clocks a warp; two Newton steps from the hardware's 20-bit FP64 reciprocal take 4 and 71
// clocks, CUDA's square root 9 and 145. Compared on 8.6e9 arguments over the whole range: the
// bits of __dsqrt_rn always, those of __drcp_rn but for mantissas of 53 ones (a tie to 2^-106,
// where the two-step form rounds down too).
//
// seed_value: the double (y0 + v 2^-44) 2^-k for a float y0 in [1/2, 1], |v| < 2^22 and
// sub = k << 20.
__device__ __forceinline__ double seed_value(float y0, int v, int sub) {
  const unsigned b = (unsigned)__float_as_int(y0);
  const unsigned long long y =
      ((unsigned long long)((b >> 3) + (896u << 20)) << 32 | (b << 29)) + (unsigned long long)(long long)(v * 512);
  return __hiloint2double((int)(y >> 32) - sub, (int)(unsigned)y);
}
// the 29 mantissa bits of a double below its leading 24, cut to 23, as a float in [0, 1) 2^s
// for the float exponent bits eb = (127 + s) << 23
__device__ __forceinline__ float low_bits(unsigned lo, int eb) {
  return __fsub_rn(__int_as_float((int)((lo >> 6) & 0x7fffffu) | eb), __int_as_float(eb));
}
constexpr float kSeedMagic = 12582912.0f;  // 1.5 2^23: the low mantissa bits of x + this are x as an integer

// 1/x for |x| in [2^-1021, 2^1021); other x take __drcp_rn
__device__ __forceinline__ double rcp(double x) {
  const int hi = __double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x);
  if ((unsigned)((hi & 0x7fffffff) - 0x00200000) >= 0x7fa00000u) return __drcp_rn(x);
  const float xh = __int_as_float((int)(__funnelshift_l(lo, (unsigned)hi, 3) & 0x7fffffu) | 0x3f800000);
  const float xl = low_bits(lo, 0x3f800000);
  float y0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(xh));
  float e = __fmaf_rn(-xh, y0, 1.0f);
  e = __fmaf_rn(__fmul_rn(y0, -0x1p-23f), xl, e);  // 1 - x y0
  const int v = __float_as_int(__fmaf_rn(__fmul_rn(y0, 0x1p44f), e, kSeedMagic)) - 0x4b400000;
  double y = seed_value(y0, v, (hi & 0x7ff00000) - (1023 << 20));
  y = __hiloint2double(__double2hiint(y) | (hi & (int)0x80000000), __double2loint(y));
  return __fma_rn(y, __fma_rn(-x, y, 1.0), y);
}

// sqrt(x) for x in [2^-900, 2^900]; other x take __dsqrt_rn
__device__ __forceinline__ double sqrt_rn(double x) {
  const int hi = __double2hiint(x);
  const unsigned lo = (unsigned)__double2loint(x);
  if ((unsigned)(hi - (123 << 20)) >= (1800u << 20)) return __dsqrt_rn(x);
  // x = m 4^k with m in [1, 4)
  const int mb = (int)((__funnelshift_l(lo, (unsigned)hi, 3) & 0xffffffu) ^ 0x800000u) + 0x3f800000;
  const float xh = __int_as_float(mb), xl = low_bits(lo, mb & 0x7f800000);
  const int k20 = ((hi - (1023 << 20)) >> 1) & (int)0xfff00000;  // k << 20
  float y0;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(xh));
  const float th = __fmul_rn(y0, y0), tl = __fmaf_rn(y0, y0, -th);
  float e = __fmaf_rn(-xh, th, 1.0f);
  e = __fmaf_rn(-xh, tl, e);
  e = __fmaf_rn(__fmul_rn(th, -0x1p-23f), xl, e);  // 1 - m y0^2
  const int v = __float_as_int(__fmaf_rn(__fmul_rn(y0, 0x1p43f), e, kSeedMagic)) - 0x4b400000;
  const double y = seed_value(y0, v, k20);
  const double g = __dmul_rn(x, y);
  const double h = __hiloint2double(__double2hiint(y) - (1 << 20), __double2loint(y));
  return __fma_rn(__fma_rn(-g, g, x), h, g);
}

// a/b, correctly rounded: with y = 1/b correctly rounded, q = a y and one residual step give the
// rounded quotient (Markstein, IBM J. Res. Dev. 34 (1990) 111). 5 FP64 operations against 9
// for the operator. a and b in [2^-255, 2^255] in magnitude (or a = 0); other arguments, and b
// with a mantissa of 53 ones (whose reciprocal rcp may round down), take the operator.
__device__ __forceinline__ double div_rn(double a, double b) {
  const int ah = __double2hiint(a), bh = __double2hiint(b);
  const unsigned ea = (unsigned)(ah & 0x7ff00000) - (768u << 20), eb = (unsigned)(bh & 0x7ff00000) - (768u << 20);
  const bool ones = (bh & 0xfffff) == 0xfffff && __double2loint(b) == -1;
  if (ea > (510u << 20) || eb > (510u << 20) || ones) {
    // a = +-0 over a finite normal b: the signed zero
    if (((ah & 0x7fffffff) | __double2loint(a)) == 0 && eb <= (510u << 20))
      return __hiloint2double((ah ^ bh) & (int)0x80000000, 0);
    return __ddiv_rn(a, b);
  }
  const double y = rcp(b), q = __dmul_rn(a, y);
  return __fma_rn(__fma_rn(-b, q, a), y, q);
}

// Natural logarithm by the table-driven method of P. T. P. Tang ("Table-driven implementation
// of the logarithm function in IEEE floating-point arithmetic", ACM TOMS 16(4), 1990):
// x = 2^k m with m in [sqrt(1/2), sqrt(2)), F = m rounded to a multiple of 1/256 (table
// entry j), r = (m - F) / F (m - F exact), log x = k log 2 + log F + log(1 + r), the last
// by its Taylor polynomial to r^6 (|r| < 2^-8.5: the omitted terms are below 2^-56 of the
// result). 15 FP64 instructions against 31 for log(); within one unit in the last place of
// the correctly rounded value (checked against an extended-precision log on 4M arguments
// from 1e-9 to 2e8 and around 1), like log(). Positive normal finite x; anything else
// goes to log(). HALF: log(x/2), the same bits as log_fast(0.5 x) (the halving is in the
// exponent).
// Tab holds the table (OpTable or LineOps: logtab, ln2_hi, ln2_lo).
template <bool HALF = false, class Tab>
__device__ __forceinline__ double log_fast(double x, const Tab& op) {
  const long long b = __double_as_longlong(x);
  if ((unsigned long long)(b - (HALF ? 0x0020000000000000LL : 0x0010000000000000LL)) >=
      (HALF ? 0x7fd0000000000000ULL : 0x7fe0000000000000ULL))
    return log(HALF ? 0.5 * x : x);
  long long k = (b >> 52) - (HALF ? 1024 : 1023);
  long long mb = (b & 0x000fffffffffffffLL) | 0x3ff0000000000000LL;  // m in [1, 2)
  if (((mb >> 44) & 0xff) >= 106) {  // m >= 1 + 106/256: use m/2 in [0.707, 1)
    mb -= 0x0010000000000000LL;
    k += 1;
  }
  const double m = __longlong_as_double(mb);
  // F = m rounded to a multiple of 2^-8, on the integer pipe: the exponent field is 1023 (m in
  // [1, sqrt 2)) or 1022
  const int mh = (int)(mb >> 32), sh = 13 - (mh >> 20 & 1);
  const int Fh = ((mh >> (sh - 1)) + 1) >> 1;  // F in units of 2^-7 or 2^-8 above its binade
  const double F = __hiloint2double(Fh << sh, 0);
  const int j = Fh - (sh == 12 ? (0x3ff00000 >> 12) - 256 : (0x3fe00000 >> 13) - 128);
  const double* T = op.logtab[j - kLogTabLo];
  const double r = (m - F) * T[0];
  double q = fma(r, -1.0 / 6.0, 1.0 / 5.0);
  q = fma(q, r, -0.25);
  q = fma(q, r, 1.0 / 3.0);
  q = fma(q, r, -0.5);
  const double p = fma(r * r, q, r);
  // (double)k without a conversion: 1.5 2^52 + k in the bits of 1.5 2^52, minus 1.5 2^52
  const double kd = __longlong_as_double(0x4338000000000000LL + k) - 0x1.8p52;
  const double hi = fma(kd, op.ln2_hi, T[1]);
  const double lo = fma(kd, op.ln2_lo, T[2]);
  return hi + (p + lo);
}

// exp(h + l) for |h| < 700 and |l| < 0.001, by the table-driven method of P. T. P. Tang
// ("Table-driven implementation of the exponential function in IEEE floating-point arithmetic",
// ACM TOMS 15(2), 1989): h + l = (128 e + j) log 2 / 128 + r with |r| < 0.0028, the result is
// 2^e (T_j + T_j (exp r - 1)) with T_j = 2^(j/128) in two parts and the Taylor polynomial of
// exp r - 1 to r^5 (the next term is below 2^-57.6 with the largest l, 2^-60 with none).
template <class Tab>
__device__ __forceinline__ double exp_parts(double h, double l, const Tab& op) {
  const double t = __fma_rn(h, op.exp_inv, 0x1.8p52);
  const int k = __double2loint(t);
  const double kd = __dsub_rn(t, 0x1.8p52);
  double r = __fma_rn(-kd, op.exp_hi, h);
  r = __dadd_rn(__fma_rn(-kd, op.exp_lo, r), l);
  double q = __fma_rn(r, 1.0 / 120.0, 1.0 / 24.0);
  q = __fma_rn(q, r, 1.0 / 6.0);
  q = __fma_rn(q, r, 0.5);
  const double p = __fma_rn(__dmul_rn(r, r), q, r);
  const double* T = op.exptab[k & 127];
  const double v = __dadd_rn(T[0], __fma_rn(T[0], p, T[1]));
  return __hiloint2double(__double2hiint(v) + ((k >> 7) << 20), __double2loint(v));
}
// exp(x): 12 FP64 operations against 19 for exp(); |x| >= 700 and NaN take exp()
template <class Tab>
__device__ __forceinline__ double exp_fast(double x, const Tab& op) {
  if ((unsigned)(__double2hiint(x) & 0x7fffffff) >= 0x4085e000u) return exp(x);
  return exp_parts(x, 0.0, op);
}

// x^y as exp(y log x), with log x in two parts from the table of log_fast (its r = (m - F)/F is
// accurate to 2^-60.5, and so are the parts), the product in two parts, and exp_parts:
// 0.5 + |y| 2^-7.5 ulp, 33 FP64 operations against 86 for pow(), which takes 1.3 ulp. x positive
// and normal with |y log x| < 700, |y| < 128 (where |y| 2^-18 of the second part stays well
// within exp_parts' polynomial, and the error below pow's); other arguments take pow().
template <class Tab>
__device__ __forceinline__ double pow_fast(double x, double y, const Tab& op) {
  const long long b = __double_as_longlong(x);
  if ((unsigned long long)(b - 0x0010000000000000LL) >= 0x7fe0000000000000ULL ||
      (unsigned)(__double2hiint(y) & 0x7fffffff) >= 0x40600000u)
    return pow(x, y);
  long long k = (b >> 52) - 1023;
  long long mb = (b & 0x000fffffffffffffLL) | 0x3ff0000000000000LL;
  if (((mb >> 44) & 0xff) >= 106) {
    mb -= 0x0010000000000000LL;
    k += 1;
  }
  const int mh = (int)(mb >> 32), sh = 13 - (mh >> 20 & 1);
  const int Fh = ((mh >> (sh - 1)) + 1) >> 1;
  const double F = __hiloint2double(Fh << sh, 0);
  const int j = Fh - (sh == 12 ? (0x3ff00000 >> 12) - 256 : (0x3fe00000 >> 13) - 128);
  const double* T = op.logtab[j - kLogTabLo];
  const double r = __dmul_rn(__dsub_rn(__longlong_as_double(mb), F), T[0]);
  const double kd = __dsub_rn(__longlong_as_double(0x4338000000000000LL + k), 0x1.8p52);
  const double hi = __fma_rn(kd, op.ln2_hi, T[3]);          // exact
  const double s = __dadd_rn(hi, r);                        // |hi| >= |r| or hi = 0
  const double e = __dadd_rn(__dsub_rn(hi, s), r);          // its rounding
  double q = __fma_rn(r, -1.0 / 6.0, 1.0 / 5.0);
  q = __fma_rn(q, r, -0.25);
  q = __fma_rn(q, r, 1.0 / 3.0);
  const double r2 = __dmul_rn(r, r);
  const double p = __fma_rn(__dmul_rn(r2, r), q, __dmul_rn(-0.5, r2));
  const double lo = __dadd_rn(__dadd_rn(p, e), __fma_rn(kd, op.ln2_lo, T[4]));
  const double h = __dmul_rn(y, s);
  const double l = __fma_rn(y, lo, __fma_rn(y, s, -h));
  if ((unsigned)(__double2hiint(h) & 0x7fffffff) >= 0x4085e000u) return pow(x, y);
  return exp_parts(h, l, op);
}

}  // namespace p2de
