// clm_math.h — table-driven log/exp/pow/log10, and sin and acos, in binary64 for C and CUDA alike.
//
// Method: P. T. P. Tang's table-driven algorithms ("Table-driven implementation of
// the exponential function in IEEE floating-point arithmetic", ACM TOMS 15(2),
// 1989, and "... the logarithm function", ACM TOMS 16(4), 1990), with Taylor
// polynomials of log1p and expm1 on the reduced argument.  The tables and split
// constants are generated by gen_math_tables.py (clm_math_tables.h).
//
// Every operation is an IEEE-754 binary64 add, multiply or fused multiply-add
// written out explicitly (CUDA: __dadd_rn/__dmul_rn/__fma_rn; C: +, *, fma() built
// with -ffp-contract=off), so a C build and a CUDA build return the same bits.  The CUDA
// build forms division, pow and log10 on the integer pipes, with the same bits (below).
//
// pow and log10 go through a double-double logarithm (cm_log_dd: Tang's table with an
// extra-precision log(c) and an exactly formed reduced argument, the error-free sums
// written out) and an exponential of a double-double argument (cm_exp_dd, 256-entry
// table in two parts), so y*log(x) keeps about 2^-67 of absolute accuracy and the
// result is rounded once at the end: nearly always the correctly rounded value, as
// Julia's own Float64 ^ (base/math.jl, double-double log and exp) nearly always is.
// Integral y in [-4096, 24576] takes Julia's compensated power by squaring instead
// (Base.Math.pow_body(x::Float64, n::Integer)), as Julia's ^ does.
//
// Accuracy (tests/test_math.py checks these against 200-bit mpmath):
//   cm_log:           absolute error below 1 ulp of max(1, |result|)
//   cm_log10:         below 0.51 ulp of max(2^-10, |result|) (double-double log)
//   cm_exp:           relative error below 2 ulp
//   cm_pow(x, y):     relative error below 0.51 ulp off the integral-y path (below 1 ulp on it);
//                     the correctly rounded value in all but a few in 10^4 random cases
//   cm_sin:           error below 1 ulp of max(|result|, 2^-53 |x|) for |x| < 2^20 pi/2
//   cm_acos:          error below 1.5 ulp on [-1, 1]
//                     (Cody-Waite reduction; the 2^-53 |x| term covers x near multiples of pi)
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define CM_FN static __device__ __forceinline__
#define CM_TABLE(name, n) static __device__ const double name[n]
#define CM_TABLE_OF(type, name, n) static __device__ const type name[n]
#define CM_LD(p) __ldg(&(p))
#define CM_FMA(a, b, c) __fma_rn((a), (b), (c))
#define CM_MUL(a, b) __dmul_rn((a), (b))
#define CM_ADD(a, b) __dadd_rn((a), (b))
#define CM_SUB(a, b) __dsub_rn((a), (b))
#define CM_SQRT(a) __dsqrt_rn(a)
#define CM_DIV(a, b) __ddiv_rn((a), (b))
#define CM_ISFINITE(x) isfinite(x)
#define CM_AS_U64(x) ((uint64_t)__double_as_longlong(x))
#define CM_AS_F64(u) __longlong_as_double((long long)(u))
#define CM_INF __longlong_as_double(0x7ff0000000000000LL)
#define CM_NAN __longlong_as_double(0x7ff8000000000000LL)
#else
#include <math.h>
#include <stdbool.h>
#include <string.h>
#define CM_FN static inline
#define CM_TABLE(name, n) static const double name[n]
#define CM_TABLE_OF(type, name, n) static const type name[n]
#define CM_LD(p) (p)
#define CM_FMA(a, b, c) fma((a), (b), (c))
#define CM_MUL(a, b) ((a) * (b))
#define CM_ADD(a, b) ((a) + (b))
#define CM_SUB(a, b) ((a) - (b))
#define CM_SQRT(a) sqrt(a)
#define CM_DIV(a, b) ((a) / (b))
#define CM_ISFINITE(x) isfinite(x)
static inline uint64_t cm_as_u64_(double x) { uint64_t u; memcpy(&u, &x, 8); return u; }
static inline double cm_as_f64_(uint64_t u) { double x; memcpy(&x, &u, 8); return x; }
#define CM_AS_U64(x) cm_as_u64_(x)
#define CM_AS_F64(u) cm_as_f64_(u)
#define CM_INF cm_as_f64_(0x7ff0000000000000ULL)
#define CM_NAN cm_as_f64_(0x7ff8000000000000ULL)
#endif

#include "clm_math_tables.h"

// ---- binary64 division on the integer pipes ----
// The correctly rounded quotient x / y formed with integer arithmetic: on GB300 an FP64
// instruction holds its sub-partition's FP64 unit for about 65 cycles (half a lane per
// clock) while a 32-bit integer multiply-add takes about 2, so a division done in
// integers leaves the FP64 unit, which bounds the column kernels, to the rest of the
// arithmetic.  Method: very-high-radix long division with quotient digits from a short
// reciprocal (D. Wong and M. Flynn, "Fast division using accurate quotient
// approximations to reduce the number of iterations", IEEE Trans. Computers 41(8),
// 1992).  With the 53-bit significands X (doubled when below Y, so that X/Y lies in
// [1, 2)) and Y:
//   R        an underestimate of 2^83 / Y, from a single-precision reciprocal of Y's
//            leading 24 bits: 0 <= 2^83/Y - R < 2600 (R >= 2^30 - 2600)
//   d1       floor-like 23-bit digit of X/Y, deficit below 43; the remainder
//            X 2^23 - d1 Y < 43 Y, exact modulo 2^64
//   d2       17 bits of that remainder over Y, deficit below 16
//   d3       12 bits, deficit below 1.3: X 2^52 = q Y + rem with 0 <= rem < 1.3 Y
// A quotient of two 53-bit significands is never a midpoint of two neighbours, so
// q + (2 rem > Y) is the quotient rounded to nearest (for rem in [Y, 1.3 Y) as well).
// The digits are correct for any R within its bounds, so the result does not depend on
// the rounding of the single-precision reciprocal.  Zero, subnormal, infinite or NaN
// operands, and quotients below the normal range or within a binade of overflow, take
// the ordinary division (CM_DIV), so the result always equals it.  Called out of line, a
// dependent chain on GB300 measures 359 cycles a division at one warp per sub-partition
// and 147 issue cycles with four (225 and 110 inlined); the 64-bit reciprocal and 2/1
// division it replaced measured 857 and 345, the hardware division 569 and 549.
CM_FN uint64_t cm_umulhi_(uint64_t a, uint64_t b) {
#if defined(__CUDACC__)
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
CM_FN uint32_t cm_umulhi32_(uint32_t a, uint32_t b) {
#if defined(__CUDACC__)
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}

// R of a significand with the hidden bit set.  The reciprocal is taken of Y's leading
// 22 bits with the next two set, at most 3 * 2^-23 above Y / 2^52 and always above 1, so
// that it lies below 1: its fraction is R's.  The argument's distance and the
// reciprocal's error (2^-23) come to less than 1300 units of 2^-31; R is lowered by as
// much.
CM_FN uint32_t cm_div_seed_(uint64_t my) {
  const uint32_t fb = 0x3f800003u | ((uint32_t)(my >> 29) & 0x7fffffu);
#if defined(__CUDACC__)
  float g;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(g) : "f"(__uint_as_float(fb)));
  const uint32_t gb = __float_as_uint(g);
#else
  float fv, g;
  memcpy(&fv, &fb, 4);
  g = 1.0f / fv;
  uint32_t gb;
  memcpy(&gb, &g, 4);
#endif
#if defined(CM_DIV_SEED_ULPS)
  return ((gb << 7) ^ 0xC0000000u) + 128 * CM_DIV_SEED_ULPS - 1300u;   // tests: other roundings
#else
  return ((gb << 7) ^ 0xC0000000u) - 1300u;                  // 2^31 g from g's bits, g in [1/2, 1)
#endif
}

// x / y without a branch, so that independent quotients overlap; *ok is false for the
// operands and quotients named above (the value is then meaningless).
CM_FN double cm_div_fx(double x, double y, bool* ok) {
  const uint64_t bx = CM_AS_U64(x), by = CM_AS_U64(y);
  const uint32_t ex = (uint32_t)(bx >> 52) & 0x7ff, ey = (uint32_t)(by >> 52) & 0x7ff;
  const uint64_t frac = 0x000fffffffffffffULL, hidden = 0x0010000000000000ULL;
  const uint64_t mx = (bx & frac) | hidden, my = (by & frac) | hidden;
  const uint32_t lt = mx < my;
  const uint32_t e = ex - ey + 1023u - lt;                  // the quotient's exponent field
  // zero, subnormal, infinite or NaN operands; a quotient not safely normal
  *ok = (ex - 1u < 0x7feu) & (ey - 1u < 0x7feu) & (e - 1u < 0x7fdu);
  const uint64_t X = mx << lt;
  const uint32_t R = cm_div_seed_(my);
  const uint32_t d1 = cm_umulhi32_((uint32_t)(X >> 22), R) >> 6;
  uint64_t rem = (X << 23) - d1 * my;
  const uint32_t d2 = cm_umulhi32_((uint32_t)(rem >> 27), R) >> 7;
  rem = (rem << 17) - d2 * my;
  const uint32_t d3 = cm_umulhi32_((uint32_t)(rem >> 25), R) >> 14;
  rem = (rem << 12) - d3 * my;
  uint64_t m = ((uint64_t)d1 << 29) + ((uint64_t)d2 << 12) + d3;
  m += (rem << 1) > my;
  // m is in [2^52, 2^53]: its hidden bit, or the carry of a round up to 2, adds to the
  // exponent field
  return CM_AS_F64(((bx ^ by) & 0x8000000000000000ULL) + ((uint64_t)(e - 1) << 52) + m);
}

#if defined(__CUDACC__)
// out of line, so that the compiler does not run it beside every quotient
static __device__ __noinline__ double cm_div_ieee_(double x, double y) { return CM_DIV(x, y); }
#else
CM_FN double cm_div_ieee_(double x, double y) { return CM_DIV(x, y); }
#endif
CM_FN double cm_div(double x, double y) {
  bool ok;
  const double q = cm_div_fx(x, y, &ok);
  if (ok) return q;
  return cm_div_ieee_(x, y);
}

// Natural logarithm.
CM_FN double cm_log(double x) {
  uint64_t ix = CM_AS_U64(x);
  if (ix - 0x0010000000000000ULL >= 0x7ff0000000000000ULL - 0x0010000000000000ULL) {
    if (x != x) return x;                                   // NaN
    if ((ix << 1) == 0) return -CM_INF;                     // +-0
    if (ix >> 63) return CM_NAN;                            // negative
    if (ix == 0x7ff0000000000000ULL) return x;              // +Inf
    ix = CM_AS_U64(CM_MUL(x, 0x1p54)) - (54ULL << 52);      // subnormal: rescale
  }
  if (ix == 0x3ff0000000000000ULL) return 0.0;              // log(1) = 0 exactly
  // x = 2^k * z with z in [0.75, 1.5); i = table interval of z
  const uint64_t tmp = ix - 0x3fe8000000000000ULL;
  const int i = (int)((tmp >> 45) & 127);
  const int64_t k = ((int64_t)tmp) >> 52;
  const double z = CM_AS_F64(ix - (tmp & 0xfff0000000000000ULL));
  const double invc = CM_LD(CM_LOG_INVC[i]);
  const double logc = CM_LD(CM_LOG_LOGC[i]);
  const double r = CM_FMA(z, invc, -1.0);                   // |r| < 0.0039
  const double kd = (double)k;
  double q = CM_FMA(r, CM_LOG_C7, CM_LOG_C6);
  q = CM_FMA(r, q, CM_LOG_C5);
  q = CM_FMA(r, q, CM_LOG_C4);
  q = CM_FMA(r, q, CM_LOG_C3);
  q = CM_FMA(r, q, CM_LOG_C2);
  const double r2 = CM_MUL(r, r);
  const double w = CM_FMA(kd, CM_LN2_HI, logc);             // k*ln2_hi is exact
  const double lo = CM_FMA(kd, CM_LN2_LO, CM_MUL(r2, q));
  return CM_ADD(w, CM_ADD(r, lo));
}

// Exponential.
CM_FN double cm_exp(double x) {
  const uint64_t ix = CM_AS_U64(x);
  const uint32_t top = (uint32_t)(ix >> 52) & 0x7ffu;
  if (top - 0x3c9u >= 0x408u - 0x3c9u) {                   // |x| < 2^-54 or |x| >= 512 or NaN/Inf
    if (top < 0x3c9u) return CM_ADD(1.0, x);
    if (x != x) return x;
    if (x > 709.782712893383973096) return CM_INF;
    if (x < -745.1332191019412076235) return 0.0;
  }
  const double shift = 0x1.8p52;
  const double z = CM_MUL(CM_INVLN2N, x);
  double kd = CM_ADD(z, shift);
  const int64_t kk = (int64_t)(CM_AS_U64(kd) - 0x4338000000000000ULL);   // round(x*64/ln2)
  kd = CM_SUB(kd, shift);
  double r = CM_FMA(-kd, CM_LN2N_HI, x);                    // kd*hi exact (36-bit hi)
  r = CM_FMA(-kd, CM_LN2N_LO, r);                           // |r| <= ln2/128
  const int j = (int)(kk & 63);
  const int64_t n = kk >> 6;                                // floor(kk / 64)
  const double tj = CM_LD(CM_EXP_T[j]);
  double p = CM_FMA(r, CM_EXP_C6, CM_EXP_C5);
  p = CM_FMA(r, p, CM_EXP_C4);
  p = CM_FMA(r, p, CM_EXP_C3);
  p = CM_FMA(r, p, CM_EXP_C2);
  p = CM_FMA(CM_MUL(r, r), p, r);                           // expm1(r)
  const double res = CM_FMA(tj, p, tj);                     // 2^(j/64) * exp(r), in [0.99, 2.01)
  if (n >= -1020 && n <= 1020) return CM_AS_F64(CM_AS_U64(res) + ((uint64_t)n << 52));
  if (n > 0) return CM_MUL(CM_AS_F64(CM_AS_U64(res) + ((uint64_t)(n - 3) << 52)), 8.0);
  // result may be subnormal: scale to normal range first, round once at the end
  return CM_MUL(CM_AS_F64(CM_AS_U64(res) + ((uint64_t)(n + 1000) << 52)), 0x1p-1000);
}

// log(x) = hi + *lo (returned: hi) for a positive finite x, subnormals included:
// |hi + lo - log(x)| below about 2^-67 max(1, |log x|), and below 2^-67 |log x| near 1.
// The pair is not renormalised: |lo| < 2^-20 max(1, |hi|), which the callers (pow and
// log10, whose products with it are formed exactly or with a single rounding) allow.
// x = 2^k z, z in [0.75, 1.5); log(x) = k ln2 + log(1/invc) + log1p(r), r = z*invc - 1
// formed exactly by one fma (the table's invc has few fractional bits), |r| < 2^-7.
CM_FN double cm_log_dd(double x, double* lo_out) {
  uint64_t ix = CM_AS_U64(x);
  if (ix < 0x0010000000000000ULL) ix = CM_AS_U64(CM_MUL(x, 0x1p54)) - (54ULL << 52);   // subnormal
  const uint64_t tmp = ix - 0x3fe8000000000000ULL;
  const int i = (int)((tmp >> 45) & 127);
  const int64_t k = ((int64_t)tmp) >> 52;
  const double z = CM_AS_F64(ix - (tmp & 0xfff0000000000000ULL));
  const double invc = CM_LD(CM_LOGD_INVC[i]);
  const double lch = CM_LD(CM_LOGD_HI[i]);
  const double lcl = CM_LD(CM_LOGD_LO[i]);
  const double r = CM_FMA(z, invc, -1.0);                    // exact
  const double kd = (double)k;
  const double t1 = CM_FMA(kd, CM_LN2_HI, lch);              // exact: multiples of 2^-42 below 2^10
  // s + e = t1 + r exactly (Dekker's Fast2Sum: |t1| >= |r| or t1 == 0, checked by the
  // table generator for every interval)
  const double s = CM_ADD(t1, r);
  const double e = CM_SUB(r, CM_SUB(s, t1));
  // -r^2/2 = ar2 + e3 exactly
  const double ar = CM_MUL(-0.5, r);
  const double ar2 = CM_MUL(ar, r);
  const double e3 = CM_FMA(ar, r, -ar2);
  // hi + e2 = s + ar2 exactly (|s| >= |ar2|)
  const double hi = CM_ADD(s, ar2);
  const double e2 = CM_ADD(CM_SUB(s, hi), ar2);
  // r^3 (1/3 - r/4 + ... + r^6/9) = (r ar2) (-2/3 + r/2 - ...): the coefficients carry
  // the factor -2 (exact); truncation below 2^-70
  double p = CM_FMA(r, CM_LOGD_C9, CM_LOGD_C8);
  p = CM_FMA(r, p, CM_LOGD_C7);
  p = CM_FMA(r, p, CM_LOGD_C6);
  p = CM_FMA(r, p, CM_LOGD_C5);
  p = CM_FMA(r, p, CM_LOGD_C4);
  p = CM_FMA(r, p, CM_LOGD_C3);
  *lo_out = CM_ADD(CM_ADD(CM_FMA(kd, CM_LN2_LO, lcl), e), CM_FMA(CM_MUL(r, ar2), p, CM_ADD(e2, e3)));
  return hi;
}

// exp(x + xl) for |xl| <= ulp(x): the value before the final rounding is within about
// 2^-61 relative; x = k ln2/256 + r with k*hi exact, 2^(j/256) = t_hi + t_lo, expm1(r)
// by its Taylor series to r^5 on |r| <= ln2/512.
CM_FN double cm_exp_dd(double x, double xl) {
  const uint64_t ix = CM_AS_U64(x);
  const uint32_t top = (uint32_t)(ix >> 52) & 0x7ffu;
  if (top - 0x3c9u >= 0x408u - 0x3c9u) {                   // |x| < 2^-54 or |x| >= 512 or NaN/Inf
    if (top < 0x3c9u) return CM_ADD(1.0, x);
    if (x != x) return x;
    if (x > 709.782712893383973096) return CM_INF;
    if (x < -745.1332191019412076235) return 0.0;
  }
  const double shift = 0x1.8p52;
  double kd = CM_FMA(x, CM_EXPD_INVLN2N, shift);
  const int64_t kk = (int64_t)(CM_AS_U64(kd) - 0x4338000000000000ULL);   // round(x*256/ln2)
  kd = CM_SUB(kd, shift);
  double r = CM_FMA(-kd, CM_EXPD_LN2N_HI, x);               // exact
  r = CM_FMA(-kd, CM_EXPD_LN2N_LO, r);
  r = CM_ADD(r, xl);
  const int j = (int)(kk & 255);
  const int64_t n = kk >> 8;                                // floor(kk / 256)
  const double th = CM_LD(CM_EXPD_THI[j]);
  const double tl = CM_LD(CM_EXPD_TLO[j]);
  double q = CM_FMA(r, CM_EXPD_C5, CM_EXPD_C4);
  q = CM_FMA(r, q, CM_EXPD_C3);
  q = CM_FMA(r, q, CM_EXPD_C2);
  const double pm = CM_FMA(CM_MUL(r, r), q, r);             // expm1(r)
  const double res = CM_ADD(th, CM_FMA(th, pm, tl));        // 2^(j/256) exp(r), in [0.99, 2.01)
  if (n >= -1020 && n <= 1020) return CM_AS_F64(CM_AS_U64(res) + ((uint64_t)n << 52));
  if (n > 0) return CM_MUL(CM_AS_F64(CM_AS_U64(res) + ((uint64_t)(n - 3) << 52)), 8.0);
  return CM_MUL(CM_AS_F64(CM_AS_U64(res) + ((uint64_t)(n + 1000) << 52)), 0x1p-1000);
}

// Julia's x^n for an integer n (Base.Math.pow_body(x::Float64, n::Integer)): power by
// squaring with the products' rounding errors carried in a second word.
CM_FN double jl_pow_int(double x, int64_t n) {
  double y = 1.0, xnlo = 0.0, ynlo = 0.0;
  if (n == 3) return CM_MUL(CM_MUL(x, x), x);
  if (n < 0) {
    const double rx = CM_DIV(1.0, x);
    if (n == -2) return CM_MUL(rx, rx);
    if (CM_ISFINITE(x)) xnlo = CM_MUL(-CM_FMA(x, rx, -1.0), rx);
    x = rx;
    n = -n;
  }
  while (n > 1) {
    if (n & 1) {
      const double err = CM_FMA(y, xnlo, CM_MUL(x, ynlo));
      const double yh = CM_MUL(x, y);
      ynlo = CM_ADD(CM_FMA(x, y, -yh), err);
      y = yh;
    }
    const double err = CM_MUL(CM_MUL(x, 2.0), xnlo);
    const double xh = CM_MUL(x, x);
    xnlo = CM_ADD(CM_FMA(x, x, -xh), err);
    x = xh;
    n >>= 1;
  }
  const double err = CM_FMA(y, xnlo, CM_MUL(x, ynlo));
  if (CM_ISFINITE(x) && CM_ISFINITE(err)) return CM_FMA(x, y, err);
  return CM_MUL(x, y);
}

// Integral y in Julia's power-by-squaring range (Base.Math.use_power_by_squaring),
// -4096 <= y <= 24576, decided on the bit pattern (integer pipes only).
CM_FN bool cm_pow_by_squaring(uint64_t uy, int64_t* n) {
  if ((uy << 1) == 0) {                                     // y = +-0
    *n = 0;
    return true;
  }
  const int ex = (int)((uy >> 52) & 0x7ff) - 1023;          // |y| in [2^ex, 2^(ex+1))
  if (ex < 0 || ex > 14) return false;                      // |y| < 1 (not 0), or |y| >= 32768
  const int sh = 52 - ex;
  const uint64_t mant = (uy & 0x000fffffffffffffULL) | 0x0010000000000000ULL;
  if (mant & ((1ULL << sh) - 1)) return false;              // a fraction
  const int64_t m = (int64_t)(mant >> sh);
  const int64_t v = (uy >> 63) ? -m : m;
  if (v < -4096 || v > 24576) return false;
  *n = v;
  return true;
}

// x^y with Julia Base's rules for Float64 (base/math.jl `^`): x == 1 -> 1; y NaN ->
// NaN; y integral in [-4096, 24576] -> compensated power by squaring (y == 0 -> 1);
// x == 0 -> 0 or Inf; x < 0 with non-integral y -> NaN (Julia raises a DomainError);
// otherwise exp(y log x) in double-double.  The tests of the common case look at bit
// patterns (integer pipes).
CM_FN double cm_pow_dd(double x, double y) {
  const uint64_t ux = CM_AS_U64(x), uy = CM_AS_U64(y);
  if (ux == 0x3ff0000000000000ULL) return 1.0;
  if ((uy << 1) > 0xffe0000000000000ULL) return y;          // y NaN
  int64_t n;
  if (cm_pow_by_squaring(uy, &n)) return n == 0 ? 1.0 : jl_pow_int(x, n);
  bool neg = false;
  if (ux - 1 >= 0x7fefffffffffffffULL) {                    // not a positive finite nonzero x
    if ((ux << 1) == 0) return y > 0.0 ? 0.0 : CM_INF;     // x = +-0
    if ((ux << 1) > 0xffe0000000000000ULL) return x;        // x NaN
    const double ay = y < 0.0 ? -y : y;
    if (ux >> 63) {                                         // x < 0
      const bool yint = ay >= 0x1p53 || (double)(int64_t)y == y;
      if (!yint) return CM_NAN;
      neg = ay < 0x1p53 && ((int64_t)y & 1);
      x = -x;
    }
    if (x == CM_INF) {
      const double v = y > 0.0 ? CM_INF : 0.0;
      return neg ? -v : v;
    }
  }
  double lxl;
  const double lxh = cm_log_dd(x, &lxl);
  const double eh = CM_MUL(y, lxh);
  const double el = CM_FMA(y, lxl, CM_FMA(y, lxh, -eh));
  const double v = cm_exp_dd(eh, el);
  return neg ? -v : v;
}

// Base-10 logarithm: the double-double log times 1/ln10 in two parts.
CM_FN double cm_log10_dd(double x) {
  const uint64_t ix = CM_AS_U64(x);
  if (ix - 0x0010000000000000ULL >= 0x7ff0000000000000ULL - 0x0010000000000000ULL) {
    if (x != x) return x;                                   // NaN
    if ((ix << 1) == 0) return -CM_INF;                     // +-0
    if (ix >> 63) return CM_NAN;                            // negative
    if (ix == 0x7ff0000000000000ULL) return x;              // +Inf
  }
  if (ix == 0x3ff0000000000000ULL) return 0.0;
  double l;
  const double h = cm_log_dd(x, &l);
  const double v = CM_MUL(h, CM_INVLN10_HI);
  const double vl = CM_ADD(CM_FMA(h, CM_INVLN10_HI, -v), CM_FMA(h, CM_INVLN10_LO, CM_MUL(l, CM_INVLN10_HI)));
  return CM_ADD(v, vl);
}

// ---- pow and log10 on the integer pipes ----
// cm_pow_dd and cm_log10_dd above take 42 and 31 FP64 instructions, 65 cycles of the FP64 unit
// each on GB300.  The same values are formed here in fixed point with 32-bit integer
// multiplies and rounded to nearest, and kept only where the rounding cannot differ from
// the FP64 functions': both are within a known distance of the true value before their
// last rounding, so when the fixed-point value lies further than the sum of the two
// distances from a midpoint of neighbouring doubles, both round to the same double.  The
// others (0.6 % of the values of pow, 0.3 % of log10 and its arguments near 1) run the
// FP64 function.  The result is therefore the FP64 function's, bit for bit (Ziv's
// rounding test: A. Ziv, "Fast evaluation of elementary mathematical functions with
// correctly rounded last bit", ACM TOMS 17(3), 1991).  Measured on GB300, a chain of
// cm_pow with 32 different lanes, cycles a call at one warp per sub-partition / issue
// cycles with four: 3,050 / 3,140 in FP64, 1,400 / 770 so (the FP64 fallback of one lane
// in some 5 calls of a warp included); cm_log10 2,170 / 2,340 and 890 / 370.
//
// log2(x) = k + log2(2^11 / C_i) + log2(1 + r), 1 + r = z C_i / 2^11 formed exactly (C_i
// of 11 bits for the 256 intervals of the significand z, r in [0, 2^-7.8)), log2(1 + r)
// its series to r^9, kept to 96 fractional bits: absolute error below 2^-71.
// 2^t, t in [0, 2^-8), by its series to t^6, times a 64-bit 2^(j/256).

// a*b >> 64 without the low partial product: at most 2 below
CM_FN uint64_t cm_umulhi_lo_(uint64_t a, uint64_t b) {
  const uint64_t ah = a >> 32, bh = b >> 32;
  const uint32_t al = (uint32_t)a, bl = (uint32_t)b;
  return ah * bh + ((ah * bl) >> 32) + ((al * bh) >> 32);
}

// |log2(x)| for the bits ix of a positive normal x, as a multiple of 2^-96 in *hi : *lo
// (128 bits); returns 1 when log2(x) is negative.
CM_FN uint32_t cm_log2_fx_(uint64_t ix, uint64_t* hi, uint64_t* lo) {
  const int64_t k = (int64_t)(ix >> 52) - 1023;
  const uint64_t m = (ix & 0x000fffffffffffffULL) | 0x0010000000000000ULL;
  const int i = (int)((ix >> 44) & 255);
  const uint64_t u = (m * (uint64_t)CM_LD(CM_FX_C[i]) - 0x8000000000000000ULL) << 8;   // r 2^7, Q64
  const uint32_t uh = (uint32_t)(u >> 32);
  uint32_t q = CM_FX_C8 - (cm_umulhi32_(uh, CM_FX_C9) >> 7);
  q = CM_FX_C7 - (cm_umulhi32_(uh, q) >> 7);
  q = CM_FX_C6 - (cm_umulhi32_(uh, q) >> 7);
  uint64_t p = CM_FX_C5 - (((uint64_t)uh * q) >> 7);
  p = CM_FX_C4 - (cm_umulhi_lo_(u, p) >> 7);
  p = CM_FX_C3 - (cm_umulhi_lo_(u, p) >> 7);
  p = CM_FX_C2 - (cm_umulhi_lo_(u, p) >> 7);
  p = CM_FX_C1 - (cm_umulhi_lo_(u, p) >> 7);                 // 1 + p = log2(1 + r) / r
  const uint64_t sl = u * p, sh = u + cm_umulhi_(u, p);      // log2(1 + r) 2^7, Q128
  const uint64_t th = CM_LD(CM_FX_LHI[i]);
  const uint64_t tl = (th << 32) | CM_LD(CM_FX_LLO[i]);
  uint64_t l = (sh << 25) | (sl >> 39);
  uint64_t h = (sh >> 39) + ((uint64_t)k << 32) + (th >> 32);
  l += tl;
  h += l < tl;
  const uint32_t neg = (uint32_t)(h >> 63);
  if (neg) {
    h = ~h + (l == 0);
    l = 0 - l;
  }
  *hi = h;
  *lo = l;
  return neg;
}

// floor(log2 v) - 48 for v >= 2^49
CM_FN int cm_top_bit_(uint64_t v) {
#if defined(__CUDACC__)
  return 15 - __clzll((long long)v);
#else
  return 15 - __builtin_clzll(v);
#endif
}

// x^y in fixed point, without a branch; false when the rounding test does not decide, or
// unless x is 1, or x is positive, normal and within 2^-60..2^60, y not an integer and
// 2^-40 <= |y| < 64, and the result safely normal.
CM_FN bool cm_pow_fx(double x, double y, double* out) {
  const uint64_t ux = CM_AS_U64(x), uy = CM_AS_U64(y);
  const uint32_t ey = (uint32_t)(uy >> 52) & 0x7ff;
  const uint64_t my = (uy << 11) | 0x8000000000000000ULL;
  const bool whole = (ey >= 1023) & (((my << 1) << ((ey - 1023) & 63)) == 0);
  const bool one = ux == 0x3ff0000000000000ULL;
  bool ok = (ux - (963ULL << 52) < (120ULL << 52)) & (ey - 983u < 46u) & !whole;
  uint64_t h, l;
  const uint32_t neg = cm_log2_fx_(ux, &h, &l) ^ (uint32_t)(uy >> 63);
  const uint64_t mh = (h << 26) | (l >> 38);                 // |log2 x| Q58, below 2^6
  const uint64_t ml = (l << 26) & 0xffffffff00000000ULL;     // its next 32 bits
  uint64_t pl = my * mh, ph = cm_umulhi_(my, mh);
  const uint64_t pe = cm_umulhi_lo_(my, ml);
  pl += pe;
  ph += pl < pe;                                             // |y log2 x| = ph:pl 2^(ey - 1023 - 121)
  const uint32_t sh = 1080u - ey;                            // 52..97
  pl = sh >= 64 ? ph : pl;
  ph = sh >= 64 ? 0 : ph;
  uint64_t n = ph >> (sh & 63);                              // integer part
  uint64_t f = ((ph << 1) << (63 - (sh & 63))) | (pl >> (sh & 63));   // fraction, Q64
  n = neg ? ~n + (f == 0) : n;
  f = neg ? 0 - f : f;
  ok &= n + 1000 < 2000;
  const int j = (int)(f >> 56);
  const uint64_t u = f << 8;                                 // t 2^8, Q64
  const uint32_t uh = (uint32_t)(u >> 32);
  uint32_t q = CM_FX_D5 + (cm_umulhi32_(uh, CM_FX_D6) >> 8);
  q = CM_FX_D4 + (cm_umulhi32_(uh, q) >> 8);                 // Q38
  uint64_t p = CM_FX_D3 + (((uint64_t)uh * q) >> 14);
  p = CM_FX_D2 + (cm_umulhi_lo_(u, p) >> 8);
  p = CM_FX_D1 + (cm_umulhi_lo_(u, p) >> 8);
  p = cm_umulhi_lo_(u, p);                                   // (2^t - 1) 2^8, Q64
  const uint64_t t = CM_LD(CM_FX_E[j]);
  const uint64_t r = t + ((cm_umulhi_lo_(t, p) + 128) >> 8);   // 2^f, Q63
  // The two values' distances from the true one, in units of 2^-63 (r in [2^63, 2^64)).
  // Here: 1/2 from the table, 1/2 from the last shift, below 0.5 from the logarithm
  // times y and the series.  cm_exp_dd: below 0.4 from its logarithm times y and its
  // series, and half a unit in the last place of each of three numbers of |argument|'s
  // binade times 2^(j/256) (the reduced argument, rounded twice, and expm1) and of the
  // product.  tm bounds the argument's magnitude / ln2, tm th8/8 the product's.  In 64ths:
  uint64_t tm = u >> 8;
  tm = (tm >> 55 ? (1ULL << 56) - tm : tm) + (1ULL << 49);
  const uint32_t th8 = (uint32_t)(t >> 60) + 1;              // 2^(j/256) < th8 / 8
  const uint64_t tw = (tm >> 3) * th8 + th8;
  const uint32_t thr = (128u + (((3u << cm_top_bit_(tm)) * th8) >> 3) + (1u << cm_top_bit_(tw))) >> 6;
  const uint32_t rest = (uint32_t)r & 0x7ff;
  const uint64_t mant = (r >> 11) + (rest >> 10);
  *out = CM_AS_F64(one ? ux : ((n + 1022) << 52) + mant);    // x == 1: 1 for every y
  return one | (ok & (rest - (0x400u - thr) > 2 * thr) & ((r >> 63) != 0));
}

// log10(x) in fixed point; false when the rounding test does not decide, x is not
// positive and normal within 2^-60..2^60, or |log10 x| < 2^-6.
CM_FN bool cm_log10_fx(double x, double* out) {
  const uint64_t ux = CM_AS_U64(x);
  if (ux - (963ULL << 52) >= (120ULL << 52)) return false;
  uint64_t h, l;
  const uint32_t neg = cm_log2_fx_(ux, &h, &l);
  const uint64_t mh = (h << 26) | (l >> 38);                 // Q58
  const uint64_t ml = (l << 26) & 0xffffffff00000000ULL;
  uint64_t pl = mh * CM_FX_LOG10_2_HI, ph = cm_umulhi_(mh, CM_FX_LOG10_2_HI);
  uint64_t pe = cm_umulhi_lo_(ml, CM_FX_LOG10_2_HI) + ((mh >> 32) * CM_FX_LOG10_2_LO);
  pl += pe;
  ph += pl < pe;                                             // Q122
  if (ph < (1ULL << 52)) return false;
#if defined(__CUDACC__)
  const int lz = __clzll((long long)ph);
#else
  const int lz = __builtin_clzll(ph);
#endif
  const uint64_t r = lz ? (ph << lz) | (pl >> (64 - lz)) : ph;
  // this value's distance from the true one is below 1 unit in the 64th place, cm_log10's
  // before its last rounding below 1/8
  const uint32_t rest = (uint32_t)r & 0x7ff;
  if (rest - 0x3feu <= 4u) return false;
  const uint64_t mant = (r >> 11) + (rest >> 10);
  *out = CM_AS_F64(((uint64_t)neg << 63) + ((uint64_t)(1027 - lz) << 52) + mant);
  return true;
}

#if defined(__CUDACC__)
// The kernels' pow and log10 (one out-of-line copy of each, and of the FP64 functions).
static __device__ __noinline__ double cm_pow_dd_call_(double x, double y) { return cm_pow_dd(x, y); }
static __device__ __noinline__ double cm_log10_dd_call_(double x) { return cm_log10_dd(x); }
CM_FN double cm_pow_inl(double x, double y) {
  double v;
  return cm_pow_fx(x, y, &v) ? v : cm_pow_dd_call_(x, y);
}
static __device__ __noinline__ double cm_pow(double x, double y) { return cm_pow_inl(x, y); }
static __device__ __noinline__ double cm_log10(double x) {
  double v;
  return cm_log10_fx(x, &v) ? v : cm_log10_dd_call_(x);
}
#else
CM_FN double cm_pow(double x, double y) { return cm_pow_dd(x, y); }
CM_FN double cm_log10(double x) { return cm_log10_dd(x); }
#endif

// sin and cos of a reduced argument r + lo, |r| <= pi/4, |lo| <= ulp(r) (Taylor
// polynomials in r^2; lo enters to first order: sin' = cos ~ 1 - r^2/2, cos' = -sin ~ -r).
CM_FN double cm_sin_poly(double r, double lo) {
  const double z = CM_MUL(r, r);
  double p = CM_FMA(z, CM_SIN_S8, CM_SIN_S7);
  p = CM_FMA(z, p, CM_SIN_S6);
  p = CM_FMA(z, p, CM_SIN_S5);
  p = CM_FMA(z, p, CM_SIN_S4);
  p = CM_FMA(z, p, CM_SIN_S3);
  p = CM_FMA(z, p, CM_SIN_S2);
  p = CM_FMA(z, p, CM_SIN_S1);
  const double lo1 = CM_FMA(CM_MUL(-0.5, z), lo, lo);       // lo (1 - r^2/2)
  return CM_ADD(r, CM_FMA(CM_MUL(r, z), p, lo1));            // r + (r^3 p + lo1)
}
CM_FN double cm_cos_poly(double r, double lo) {
  const double z = CM_MUL(r, r);
  double q = CM_FMA(z, CM_COS_C8, CM_COS_C7);
  q = CM_FMA(z, q, CM_COS_C6);
  q = CM_FMA(z, q, CM_COS_C5);
  q = CM_FMA(z, q, CM_COS_C4);
  q = CM_FMA(z, q, CM_COS_C3);
  q = CM_FMA(z, q, CM_COS_C2);
  // 1 - z/2 + z^2 q - r lo, with the rounding error of w = 1 - z/2 carried into the tail
  const double hz = CM_MUL(0.5, z);
  const double w = CM_SUB(1.0, hz);
  const double c = CM_FMA(-r, lo, CM_SUB(CM_SUB(1.0, w), hz));
  return CM_ADD(w, CM_FMA(CM_MUL(z, z), q, c));
}

// Sine for |x| < 2^20 * pi/2 (NaN beyond, and for NaN or infinite x): the reduced
// argument x - k pi/2 = r + lo with pi/2 in three parts (k*hi and k*mid exact, the
// subtraction of k*mid error-free by Knuth's two-sum), then sin or cos by k mod 4.
CM_FN double cm_sin(double x) {
  const double ax = x < 0.0 ? -x : x;
  if (!(ax < 1647099.0)) return CM_NAN;                     // 2^20 * pi/2, NaN, Inf
  if (ax < 0x1p-27) return x;                               // sin(x) = x in binary64
  if (ax <= CM_PIO4) return cm_sin_poly(x, 0.0);
  const double shift = 0x1.8p52;
  double kd = CM_FMA(x, CM_INVPIO2, shift);
  const int64_t k = (int64_t)(CM_AS_U64(kd) - 0x4338000000000000ULL);   // round(x*2/pi)
  kd = CM_SUB(kd, shift);
  const double a = CM_FMA(-kd, CM_PIO2_HI, x);              // exact
  const double b = CM_MUL(-kd, CM_PIO2_MID);                // exact
  const double r0 = CM_ADD(a, b);
  const double bv = CM_SUB(r0, a);
  const double err = CM_ADD(CM_SUB(a, CM_SUB(r0, bv)), CM_SUB(b, bv));   // a + b - r0
  const double lo0 = CM_FMA(-kd, CM_PIO2_LO, err);
  const double r = CM_ADD(r0, lo0);
  const double lo = CM_SUB(lo0, CM_SUB(r, r0));
  const int q = (int)(k & 3);
  const double v = (q & 1) ? cm_cos_poly(r, lo) : cm_sin_poly(r, lo);
  return (q & 2) ? -v : v;
}

// asin(t) for |t| <= 1/2: t + t^3 P(t^2) (Taylor series, 27 terms).
CM_FN double cm_asin_small(double t) {
  const double z = CM_MUL(t, t);
  double p = CM_ASIN_A27;
  p = CM_FMA(z, p, CM_ASIN_A26);
  p = CM_FMA(z, p, CM_ASIN_A25);
  p = CM_FMA(z, p, CM_ASIN_A24);
  p = CM_FMA(z, p, CM_ASIN_A23);
  p = CM_FMA(z, p, CM_ASIN_A22);
  p = CM_FMA(z, p, CM_ASIN_A21);
  p = CM_FMA(z, p, CM_ASIN_A20);
  p = CM_FMA(z, p, CM_ASIN_A19);
  p = CM_FMA(z, p, CM_ASIN_A18);
  p = CM_FMA(z, p, CM_ASIN_A17);
  p = CM_FMA(z, p, CM_ASIN_A16);
  p = CM_FMA(z, p, CM_ASIN_A15);
  p = CM_FMA(z, p, CM_ASIN_A14);
  p = CM_FMA(z, p, CM_ASIN_A13);
  p = CM_FMA(z, p, CM_ASIN_A12);
  p = CM_FMA(z, p, CM_ASIN_A11);
  p = CM_FMA(z, p, CM_ASIN_A10);
  p = CM_FMA(z, p, CM_ASIN_A9);
  p = CM_FMA(z, p, CM_ASIN_A8);
  p = CM_FMA(z, p, CM_ASIN_A7);
  p = CM_FMA(z, p, CM_ASIN_A6);
  p = CM_FMA(z, p, CM_ASIN_A5);
  p = CM_FMA(z, p, CM_ASIN_A4);
  p = CM_FMA(z, p, CM_ASIN_A3);
  p = CM_FMA(z, p, CM_ASIN_A2);
  p = CM_FMA(z, p, CM_ASIN_A1);
  return CM_FMA(CM_MUL(t, z), p, t);
}

// Arc cosine for |x| <= 1 (NaN outside): pi/2 - asin(x) on |x| <= 1/2, else through
// asin(sqrt((1 -+ x)/2)), whose argument is formed exactly ((1 -+ x) by Sterbenz, the
// halving) and rounded once by the square root.
CM_FN double cm_acos(double x) {
  if (!(x >= -1.0 && x <= 1.0)) return CM_NAN;
  if (x <= 0.5 && x >= -0.5) return CM_ADD(CM_PIO2_H, CM_SUB(CM_PIO2_L, cm_asin_small(x)));
  if (x > 0.5) return CM_MUL(2.0, cm_asin_small(CM_SQRT(CM_MUL(0.5, CM_SUB(1.0, x)))));
  const double a = CM_MUL(2.0, cm_asin_small(CM_SQRT(CM_MUL(0.5, CM_ADD(1.0, x)))));
  return CM_ADD(CM_PI_HI, CM_SUB(CM_PI_LO, a));
}
