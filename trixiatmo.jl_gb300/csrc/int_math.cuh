// Reciprocals, roots, logarithms, exponentials and logarithmic means of FP64
// values on the integer pipe.
//
// Why: GB300 issues 2 FP64 operations per SM and clock (a measured DFMA stream
// reaches 1.57), but 128 32-bit ones; a warp's FP64 instruction takes the pipe
// for 16 cycles, in which four sub-partitions issue 64 others.  With CUDA's FP64
// functions the element and interface kernels kept that pipe 75-89 % busy and
// issued only 6-11 instructions per FP64 one.  Measured in FP64-operation times on this chip,
// 1/x costs 4.5, a/b 7.1, sqrt 7.5, rsqrt 4.7, exp 16, log 31 and pow 78; the
// forms below take the FP64 pipe for none of them.  The integer pipe multiplies
// 32 x 32 -> 64 bits at 22 per SM and clock: a 64-bit high product costs 0.2
// FP64 operations.
//
// Numbers are fixed-point words (Qi.f: i integer and f fraction bits) of the
// significands, so every result carries about 60 bits before its one rounding
// to 53: errors are below 0.52 ulp (rcp, sqrt, rsqrt, div) and 0.6 ulp (pow,
// means), where the FP64 sequences give 0.5 to 2.  Arguments outside the
// normal positive range (zeros, subnormals, infinities, NaN) take the CUDA
// function in an out-of-line branch, so special values come out as before.
//
// The same code runs on the host (only the 24-bit seeds differ), where it is
// compared with exact arithmetic.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>
#include <cuda_runtime.h>

#include "int_math_tables.cuh"

#ifdef __CUDACC__
#define TAG_HD __host__ __device__ __forceinline__
#define TAG_SLOW static __host__ __device__ __noinline__
#else
#define TAG_HD inline
#define TAG_SLOW static inline
#endif

namespace tag {

using u64 = unsigned long long;
using i64 = long long;
using u32 = unsigned int;

// ---- bit access and word products -------------------------------------------
TAG_HD u64 f64_bits(double x) {
#ifdef __CUDA_ARCH__
  return (u64)__double_as_longlong(x);
#else
  u64 b;
  std::memcpy(&b, &x, 8);
  return b;
#endif
}
TAG_HD double f64_from(u64 b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((i64)b);
#else
  double x;
  std::memcpy(&x, &b, 8);
  return x;
#endif
}
TAG_HD float f32_from(u32 b) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float x;
  std::memcpy(&x, &b, 4);
  return x;
#endif
}
TAG_HD u32 f32_bits(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  u32 b;
  std::memcpy(&b, &x, 4);
  return b;
#endif
}
TAG_HD u32 mulhi32(u32 a, u32 b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (u32)(((u64)a * b) >> 32);
#endif
}
TAG_HD u64 mulhi64(u64 a, u64 b) {
#ifdef __CUDA_ARCH__
  return __umul64hi(a, b);
#else
  return (u64)(((unsigned __int128)a * b) >> 64);
#endif
}
TAG_HD i64 smulhi64(i64 a, i64 b) {
#ifdef __CUDA_ARCH__
  return __mul64hi(a, b);
#else
  return (i64)(((__int128)a * b) >> 64);
#endif
}
// High word of an unsigned product without the low words' part: the error is
// in [-3, 0] and -1.25 on average.
TAG_HD u64 umul_high(u64 a, u64 b) {
  const u32 ah = (u32)(a >> 32), al = (u32)a, bh = (u32)(b >> 32), bl = (u32)b;
  return (u64)ah * bh + mulhi32(ah, bl) + mulhi32(al, bh);
}
// (a b) >> 32 of a 64-bit and a 32-bit word
TAG_HD u64 mulhi64x32(u64 a, u32 b) {
  return (u64)(u32)(a >> 32) * b + mulhi32((u32)a, b);
}
TAG_HD int leading_zeros(u64 a) {
#ifdef __CUDA_ARCH__
  return __clzll((i64)a);
#else
  return a ? __builtin_clzll(a) : 64;
#endif
}
TAG_HD float rcp_seed(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.0f / x;
#endif
}
TAG_HD float rsqrt_seed(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.0f / sqrtf(x);
#endif
}
TAG_HD int f32_to_int(float x) {
#ifdef __CUDA_ARCH__
  return __float2int_rn(x);
#else
  return (int)lrintf(x);
#endif
}

// Exponent field of a double's high word (sign dropped) and whether it is a
// normal number; the significand 1.f as Q1.63 (top bit set).
TAG_HD u32 f64_exponent(u64 b) { return (u32)(b >> 52) & 0x7ffu; }
TAG_HD bool normal_exponent(u32 e) { return e - 1u < 0x7feu; }
TAG_HD u64 significand(u64 b) { return (b << 11) | 0x8000000000000000ull; }

// a Q0.64 or Q1.63 word to its upper 53 bits, rounded (up to 2^53)
TAG_HD u64 round53(u64 y) { return (y >> 11) + ((y >> 10) & 1u); }

// ---- reciprocal, square roots, quotient ---------------------------------------
// A binary32 seed in [1/2, 1] as Q0.32, lowered by `places` last places and
// not below the 1/2 that bounds the exact value.
TAG_HD u32 seed_q32(float r, u32 places) {
  const u32 s = f32_bits(r) - places;
  return ((s > 0x3f000000u ? s : 0x3f000000u) << 8) | 0x80000000u;
}

// 1/m of a significand m (Q1.63) as Q0.64 in (1/2, 1): a 24-bit seed from
// below, y0 <= 1/m, then y = y0 (1 + e + e^2) with the exact residual
// e = 1 - m y0 < 2^-20 (the cubic Newton step; the next term is < 2^-60).
TAG_HD u64 rcp_significand(u64 m) {
  // the seed lowered by four of its last places: m was truncated to 24 bits
  // (two places) and the hardware's reciprocal is good to one
  const u32 y0 = seed_q32(rcp_seed(f32_from(0x3f800000u | ((u32)(m >> 40) & 0x7fffffu))), 4u);
  const u64 es = ((1ull << 63) - mulhi64x32(m, y0)) << 20;         // e, Q.83
  const u64 c = mulhi64x32(es, y0);                                // y0 e, Q.83
  const u32 c2 = mulhi32((u32)(c >> 32), (u32)(es >> 32));         // y0 e^2, Q.70
  return ((u64)y0 << 32) + (c >> 19) + (c2 >> 6);
}

// 1/sqrt(a) of a in [1, 4) (Q2.62) as Q0.64 in (1/2, 1): as above with
// y = y0 (1 + e/2 + 3 e^2 / 8), e = 1 - a y0^2.
TAG_HD u64 rsqrt_significand(u64 a) {
  const u32 top = (u32)(a >> 62) > 1u;  // a >= 2: the binary32 exponent is one more
  const u32 f = top ? 0x40000000u | ((u32)(a >> 40) & 0x7fffffu)
                    : 0x3f800000u | ((u32)(a >> 39) & 0x7fffffu);
  const u32 y0 = seed_q32(rsqrt_seed(f32_from(f)), 5u);  // the seed is good to two places
  const u64 es = ((1ull << 62) - mulhi64(a, (u64)y0 * y0)) << 20;  // e, Q.82
  const u64 c = mulhi64x32(es, y0);                                // y0 e, Q.82
  const u32 c2 = mulhi32((u32)(c >> 32), (u32)(es >> 32));         // y0 e^2, Q.68
  return ((u64)y0 << 32) + (c >> 19) + ((3ull * c2) >> 7);
}

TAG_SLOW double slow_rcp(double x) { return 1.0 / x; }
TAG_SLOW double slow_div(double a, double b) { return a / b; }
TAG_SLOW double slow_sqrt(double x) { return sqrt(x); }
TAG_SLOW double slow_rsqrt(double x) { return 1.0 / sqrt(x); }

// 1/x.  The packed exponent is one less and the significand's leading bit is
// added to it, so a round-up to the next power of two carries by itself.
TAG_HD double int_rcp(double x) {
  const u64 b = f64_bits(x);
  const u32 e = f64_exponent(b);
  if (e - 1u >= 2044u) return slow_rcp(x);  // 1/x would be subnormal from e = 2045
  const u64 y = rcp_significand(significand(b));
  return f64_from((b & 0x8000000000000000ull) | (((u64)(2044u - e) << 52) + round53(y)));
}

// a/b with one rounding: the product of a's significand and 1/b's.
TAG_HD double int_div(double a, double b) {
  const u64 ba = f64_bits(a), bb = f64_bits(b);
  const u32 ea = f64_exponent(ba), eb = f64_exponent(bb);
  const int e = (int)ea - (int)eb + 1023;
  if (!normal_exponent(ea) || !normal_exponent(eb) || e < 2 || e > 2045) return slow_div(a, b);
  u64 q = mulhi64(significand(ba), rcp_significand(significand(bb)));  // Q1.63, in (1/2, 2)
  const int low = (int)(q >> 63) ^ 1;                                  // quotient below 1
  q <<= low;
  return f64_from(((ba ^ bb) & 0x8000000000000000ull) |
                  (((u64)(e - low - 1) << 52) + round53(q)));
}

// a in [1, 4) (Q2.62) with x = a 2^(2k), from the bits of a normal positive x
TAG_HD u64 even_significand(u64 b, u32 e, int& k) {
  const int t = (int)e - 1023;
  k = t >> 1;
  return significand(b) >> (1 - (t & 1));
}

TAG_HD double int_sqrt(double x) {
  const u64 b = f64_bits(x);
  const u32 e = (u32)(b >> 52);  // the sign bit makes it out of range
  if (!normal_exponent(e)) return slow_sqrt(x);
  int k;
  const u64 a = even_significand(b, e, k);
  const u64 s = mulhi64(a, rsqrt_significand(a));  // Q2.62, in [1, 2)
  return f64_from(((u64)(k + 1022) << 52) + ((s + 512u) >> 10));
}

TAG_HD double int_rsqrt(double x) {
  const u64 b = f64_bits(x);
  const u32 e = (u32)(b >> 52);
  if (!normal_exponent(e)) return slow_rsqrt(x);
  int k;
  const u64 y = rsqrt_significand(even_significand(b, e, k));
  return f64_from(((u64)(1021 - k) << 52) + round53(y));
}

// ---- logarithm, exponential, power ----------------------------------------------
struct LogEntry {
  u64 t;  // -log2(y / 512), Q0.63
  u64 y;
};
#ifdef __CUDACC__
static __device__ const LogEntry kLogTableDev[128] = {TAG_LOG_TABLE};
static __device__ const u64 kExp2TableDev[128] = {TAG_EXP2_TABLE};
#endif
static const LogEntry kLogTableHost[128] = {TAG_LOG_TABLE};
static const u64 kExp2TableHost[128] = {TAG_EXP2_TABLE};

TAG_HD LogEntry log_entry(u32 i) {
#ifdef __CUDA_ARCH__
  const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(kLogTableDev) + i);
  return LogEntry{v.x, v.y};
#else
  return kLogTableHost[i];
#endif
}
TAG_HD u64 exp2_entry(u32 j) {
#ifdef __CUDA_ARCH__
  return __ldg(kExp2TableDev + j);
#else
  return kExp2TableHost[j];
#endif
}

// log2 of a significand m (Q1.63) as Q0.63 (absolute error < 2^-57): the
// table's 10-bit reciprocal y makes f = m y - 1 exact with |f| < 2^-7.6, and
// log2(1 + f) = f (c1 + f (c2 + f (c3 + f P(f)))), P in binary32.
TAG_HD i64 log2_significand(u64 m) {
  const LogEntry t = log_entry((u32)(m >> 56) & 127u);
  const i64 f = (i64)((m >> 3) * t.y);  // Q.69; 1.0 = 2^69 drops out modulo 2^64
  const float ff = (float)(int)(f >> 32) * 7.275957614183426e-12f;  // 2^-37
  const float P = fmaf(ff, fmaf(ff, fmaf(ff, TAG_LOG2_C7, TAG_LOG2_C6), TAG_LOG2_C5), TAG_LOG2_C4);
  const i64 p = (i64)f32_to_int(P * 2147483648.0f);                 // Q.31
  const i64 q3 = TAG_LOG2_C3 + (((f >> 32) * p) >> 6);              // Q.62
  const i64 q2 = TAG_LOG2_C2 + (smulhi64(f, q3) >> 5);
  const i64 q1 = TAG_LOG2_C1 + (smulhi64(f, q2) >> 5);
  return (i64)t.t + (smulhi64(f, q1) >> 4);
}

// exp2 of a fraction g (Q0.64) as a significand in [1, 2) (Q1.63): table for
// the top seven bits, 2^r - 1 = r (c1 + r (c2 + r (c3 + r P(r)))) for the rest.
TAG_HD u64 exp2_fraction(u64 g) {
  const u64 base = exp2_entry((u32)(g >> 57));
  const u64 r = g & 0x01ffffffffffffffull;                           // Q.64, < 2^-7
  const float rf = (float)(int)(r >> 32) * 2.3283064365386963e-10f;  // 2^-32
  const float P = fmaf(rf, fmaf(rf, TAG_EXP2_C6, TAG_EXP2_C5), TAG_EXP2_C4);
  const u64 p = (u64)(u32)f32_to_int(P * 17179869184.0f) << 29;      // Q.34 -> Q.63
  const u64 q3 = TAG_EXP2_C3 + mulhi64(r, p);
  const u64 q2 = TAG_EXP2_C2 + mulhi64(r, q3);
  const u64 q1 = TAG_EXP2_C1 + mulhi64(r, q2);
  return base + 2 * mulhi64(base, mulhi64(r, q1));                   // r q1: Q.63
}

TAG_SLOW i64 slow_log2_fixed(double x) {
  // Subnormals are scaled up.  Values that have no logarithm (bad states, and
  // partial densities below zero) get words that keep them out of the means'
  // series beside any other value: negative ones the word of |x| and 2^62 (1024
  // octaves), zeros -1536 octaves.  Infinities and NaN give 0; they make the
  // means non-finite by themselves.
  if (x == 0.0) return -(1536ll << 52);
  if (x != x || f64_exponent(f64_bits(x)) == 0x7ffu) return 0;
  const double m = x < 0.0 ? -x : x;
  const u64 b = f64_bits(m < 1.0 ? m * 18014398509481984.0 : m);  // 2^54
  const i64 e = (i64)f64_exponent(b) - 1023 - (m < 1.0 ? 54 : 0);
  return e * (1ll << 52) + ((log2_significand(significand(b)) + 1024) >> 11) +
         (x < 0.0 ? 1ll << 62 : 0);
}

// log2(x) as Q11.52 for normal positive x (absolute error < 2^-53): the node
// quantity that differences of logarithms are taken of.
TAG_HD i64 log2_fixed(double x) {
  const u64 b = f64_bits(x);
  const u32 e = (u32)(b >> 52);
  if (!normal_exponent(e)) return slow_log2_fixed(x);
  return ((i64)e - 1023) * (1ll << 52) + ((log2_significand(significand(b)) + 1024) >> 11);
}

// Packs 2^(i + g), g in [0, 1) as Q0.64; i must give a normal number.
TAG_HD double pack_exp2(int i, u64 g) {
  return f64_from(((u64)(i + 1022) << 52) + round53(exp2_fraction(g)));
}

TAG_SLOW double slow_pow(double x, double y) { return pow(x, y); }
TAG_SLOW double slow_exp(double x) { return exp(x); }

// x^y from y as a word with F fraction bits (below 2^63), for normal x whose
// power is normal too; ok is cleared otherwise.  y log2 x = y t + y l with t the
// exponent and l the log2 of the significand.
template <int F>
TAG_HD double int_pow_word(double x, u64 yq, bool& ok) {
  const u64 b = f64_bits(x);
  const u32 e = (u32)(b >> 52);
  ok = normal_exponent(e) && yq != 0;
  const i64 t = (i64)e - 1023;
  i64 l = log2_significand(significand(b));                  // Q.63
  l = l < 0 ? 0 : l;
  const u64 yl = mulhi64(yq, (u64)l << 1);                   // y l, Q.F
  const i64 ti = smulhi64(t << (64 - F), (i64)yq);           // floor(y t)
  const u64 tf = ((u64)(t << (64 - F)) * yq) >> (64 - F);    // its fraction, Q.F
  const u64 s = tf + yl;
  const int i = (int)ti + (int)(s >> F);
  ok = ok && i >= -1020 && i <= 1020;
  return pack_exp2(ok ? i : 0, s << (64 - F));
}

// An exponent y in (0, 4) as Q2.61 for int_pow; 0 (the out-of-line branch)
// for any other.
inline u64 pow_exponent(double y) {
  return y > 0.0 && y < 4.0 ? (u64)(y * 2305843009213693952.0) : 0;
}

// x^y for a fixed exponent y (a ratio of gas constants), y_q61 = pow_exponent(y).
TAG_HD double int_pow(double x, double y, u64 y_q61) {
  bool ok;
  const double r = int_pow_word<61>(x, y_q61, ok);
  return ok ? r : slow_pow(x, y);
}

// x^y for an exponent in [1/64, 16), which Q4.58 holds exactly.
TAG_HD double int_pow(double x, double y) {
  const u64 b = f64_bits(y);
  const int sh = (int)(b >> 52) - 1023;
  bool ok = sh >= -6 && sh <= 3;
  const double r = int_pow_word<58>(x, ok ? (significand(b) >> 5) >> -(sh < 0 ? sh : 0) << (sh > 0 ? sh : 0) : 0, ok);
  return ok ? r : slow_pow(x, y);
}

// e^x for |x| < 512: x log2 e in fixed point, its integer part the exponent.
TAG_HD double int_exp(double x) {
  const u64 b = f64_bits(x);
  const u32 e = f64_exponent(b);
  if (e >= 1032u) return slow_exp(x);  // |x| >= 512, infinities, NaN
  // |x| as Q4.60 below 16, else as Q10.54 (tiny values shift out: e^x rounds
  // to 1), times log2 e as Q2.62: the high word Q6.58 or Q12.52 and 64 more bits
  const int sh = (int)e - 1023, up = sh < 4 ? 3 : 9;
  const u64 m = significand(b) >> up;
  const u64 a = sh >= 0 ? m << sh : (sh > -63 ? m >> -sh : 0);
  const u64 hi = mulhi64(a, TAG_LOG2E_Q62), lo = a * (u64)TAG_LOG2E_Q62;
  u64 g = (hi << (up + 3)) | (lo >> (61 - up));  // fraction, Q0.64
  int i = (int)(hi >> (61 - up));
  if ((i64)b < 0) {
    g = 0 - g;
    i = -i - (g != 0);
  }
  return pack_exp2(i, g);
}

TAG_SLOW double slow_log2_ratio(double x, i64 ref_q58) {
  return log2(x) - (double)ref_q58 * 3.469446951953614e-18;  // 2^-58
}

// log2(x) - ref for a reference in [-8, 8] given as ref 2^58 rounded; absolute
// error 2^-57 for x within 2^+-15 (one rounding of the result besides).
TAG_HD double int_log2_ratio(double x, i64 ref_q58) {
  const u64 b = f64_bits(x);
  const int t = (int)(b >> 52) - 1023;
  if (t < -15 || t > 14) return slow_log2_ratio(x, ref_q58);
  const i64 v = (i64)t * (1ll << 58) + (log2_significand(significand(b)) >> 5) - ref_q58;
  return (double)v * 3.469446951953614e-18;  // 2^-58
}

// ---- means ------------------------------------------------------------------------
// z = d^2 (Q0.64) of a difference d of two log2_fixed values, |d| < 1 (values
// within a factor of two); series_in_range tests it for one or two differences
// by the OR of their magnitudes.
TAG_HD u64 magnitude(i64 d) { return d < 0 ? 0ull - (u64)d : (u64)d; }
TAG_HD bool series_in_range(u64 a) { return (u32)(a >> 32) < (1u << 20); }
TAG_HD u64 log_square(u64 a) { return umul_high(a << 12, a << 12); }

// 1 - c for c (Q0.64) below 1/2, rounded to 53 bits: numbers just below 1 are
// spaced by 2^-53, so the subtraction is one of the bit patterns.
TAG_HD double one_minus(u64 c) { return f64_from(0x3ff0000000000000ull - ((c + 1024u) >> 11)); }

// 1 - tanh(x)/x (Q0.64) at x = d ln2 / 2: ln_mean(u, v) = (u + v)/2 tanh(x)/x, with
// d = log2(v) - log2(u) (ln_mean = (u + v)/2 t/atanh(t) and t = tanh(x)).
// Taylor series in z, the first seven terms in integers, six more in binary32
// (below 2^-35 together).  No reciprocal and no branch on the size of d.
TAG_HD u64 ln_mean_deficit(u64 z) {
  const float zf = (float)(u32)(z >> 32) * 2.3283064365386963e-10f;
  const float P = fmaf(zf, -fmaf(zf, -fmaf(zf, -fmaf(zf, -TAG_LN_B4, TAG_LN_B3), TAG_LN_B2),
                                 TAG_LN_B1), TAG_LN_B0);
  // the small coefficients in 32-bit words (the tail and A6 in Q.61, the product
  // under A4 in Q.56): below 2^-57 of the result at z = 1
  const u32 zh = (u32)(z >> 32);
  const u32 p6 = (u32)(TAG_LN_A6 >> 3) - mulhi32(zh, (u32)f32_to_int(P * 2.305843009213694e18f));
  u64 p = TAG_LN_A5 - ((u64)mulhi32(zh, p6) << 3);
  p = TAG_LN_A4 - ((u64)mulhi32(zh, (u32)(p >> 8)) << 8);
  p = TAG_LN_A3 - umul_high(z, p);
  p = TAG_LN_A2 - umul_high(z, p);
  p = TAG_LN_A1 - umul_high(z, p);
  p = TAG_LN_A0 - umul_high(z, p);
  return umul_high(z, p);
}

// 1 - x/sinh(x) (Q0.64) at x = d ln2: inv_ln_mean(1/u, 1/v) = (u + v)/2 x/sinh(x) (with
// r = v/u: log(r)/(1/u - 1/v) = u v log(r)/(v - u), and (u + v)(v - u)/(2 u v)
// = sinh(log r)).  So the mean of reciprocals needs no reciprocal.
TAG_HD u64 inv_ln_mean_deficit(u64 z) {
  const float zf = (float)(u32)(z >> 32) * 2.3283064365386963e-10f;
  const float P = fmaf(zf, -fmaf(zf, -fmaf(zf, -fmaf(zf, -TAG_INV_B4, TAG_INV_B3), TAG_INV_B2),
                                 TAG_INV_B1), TAG_INV_B0);
  // the small coefficients in 32-bit words (the tail and A6 in Q.61, the product
  // under A4 in Q.56): below 2^-57 of the result at z = 1
  const u32 zh = (u32)(z >> 32);
  const u32 p6 = (u32)(TAG_INV_A6 >> 3) - mulhi32(zh, (u32)f32_to_int(P * 2.305843009213694e18f));
  u64 p = TAG_INV_A5 - ((u64)mulhi32(zh, p6) << 3);
  p = TAG_INV_A4 - ((u64)mulhi32(zh, (u32)(p >> 8)) << 8);
  p = TAG_INV_A3 - umul_high(z, p);
  p = TAG_INV_A2 - umul_high(z, p);
  p = TAG_INV_A1 - umul_high(z, p);
  p = TAG_INV_A0 - umul_high(z, p);
  return umul_high(z, p);
}

// The same for z below 2^-11 (values within 1.5 %: the horizontal pairs of a
// smooth atmosphere): three terms, the inner two in 32-bit words (error below
// 2^-57); 40 instructions instead of 85.
constexpr u64 kShortZ = 1ull << 53;
TAG_HD u64 short_deficit(u64 z, u64 a0, u32 a1_q39, u32 a2_q40) {
  const u32 zn = (u32)(z >> 21);                             // z 2^11 in Q0.32
  const u32 p1 = a1_q39 - (mulhi32(zn, a2_q40) >> 12);       // a1 - z a2, Q.39
  return umul_high(z, a0 - (((u64)zn * p1) >> 18));          // a0 - z p1, Q.64
}
TAG_HD u64 ln_mean_deficit_short(u64 z) {
  return short_deficit(z, TAG_LN_A0, (u32)(TAG_LN_A1 >> 25), (u32)(TAG_LN_A2 >> 24));
}
TAG_HD u64 inv_ln_mean_deficit_short(u64 z) {
  return short_deficit(z, TAG_INV_A0, (u32)(TAG_INV_A1 >> 25), (u32)(TAG_INV_A2 >> 24));
}

TAG_HD double ln_mean_factor(u64 z) { return one_minus(ln_mean_deficit(z)); }
TAG_HD double inv_ln_mean_factor(u64 z) { return one_minus(inv_ln_mean_deficit(z)); }

// A mean's factor 1 - z (a0 + z (a1 + ...)) with coefficients of run-time
// parameters, in the same form (any signs; seven Q0.63 words, six binary32).
// ok: the fixed-point form holds (the factor stays within (1/2, 1]).
struct EvenSeries {
  i64 a[7];
  float b[6];
  int ok;
};
TAG_HD u64 even_deficit(const EvenSeries& s, u64 z) {
  const i64 zq = (i64)(z >> 1);  // Q0.63
  const float zf = (float)(u32)(z >> 32) * 2.3283064365386963e-10f;
  float P = s.b[5];
#pragma unroll
  for (int k = 4; k >= 0; --k) P = fmaf(zf, P, s.b[k]);
  i64 p = (i64)f32_to_int(P * 1.152921504606847e18f) << 3;  // Q.60 -> Q.63
#pragma unroll
  for (int k = 6; k >= 0; --k) p = s.a[k] + (smulhi64(zq, p) << 1);
  return (u64)(smulhi64(zq, p) << 2);
}
TAG_HD double even_factor(const EvenSeries& s, u64 z) { return one_minus(even_deficit(s, z)); }

// The factors beyond a factor of two between the values, up to 256: D = |d| in
// [1, 8) as a log2_fixed word.  With E = 2^-D all three means' factors are
// quotients of 1 +- E and its powers, so one to three table exponentials and a
// reciprocal of 64-bit words serve where the FP64 forms took logarithms'
// differences, divisions and, for the Stolarsky mean, two powers.  They depend
// on D alone, to which their relative sensitivity is below 1 (the absolute error
// of D is below 2^-52); relative error of the forms themselves below 2^-56.
// Right-hand side of the potential-temperature shell (flux_tec, polydeg 4,
// elements 7.5 km tall, whose end-to-end vertical pairs lie here): 285 us with
// the FP64 forms, 212 us with these.
TAG_HD bool middle_range(u64 a) { return (u32)(a >> 32) < (8u << 20); }

// 2^-q for q > 0 with F fraction bits as e 2^-k, e in [1, 2) (Q1.63).
template <int F>
TAG_HD u64 exp2_negative(u64 q, int& k) {
  k = (int)(q >> F) + ((q << (64 - F)) != 0);
  return exp2_fraction((0 - q) << (64 - F));
}
// The same as Q1.63 itself.
template <int F>
TAG_HD u64 exp2_negative(u64 q) {
  int k;
  const u64 e = exp2_negative<F>(q, k);
  return k < 64 ? e >> k : 0;
}

// 1 - tanh(x)/x, x = D ln2 / 2: tanh(x)/x = 2 (1 - E) / ((1 + E) D ln2)
TAG_HD u64 ln_mean_deficit_middle(u64 a) {
  const u64 one = 1ull << 63, E = exp2_negative<52>(a);
  const u64 x = mulhi64(a << 9, TAG_LN2_Q64);   // D ln2, Q3.61
  const u64 den = mulhi64(one + E, x);          // Q4.60, in (1, 6)
  const int lz = leading_zeros(den);
  const u64 q = mulhi64(one - E, rcp_significand(den << lz));
  return 0 - (q << (lz - 1));  // 1 <= lz <= 3
}

// 1 - x/sinh(x), x = D ln2: x/sinh(x) = 2 x E / (1 - E^2)
TAG_HD u64 inv_ln_mean_deficit_middle(u64 a) {
  int k;
  const u64 e = exp2_negative<52>(a, k), E = e >> k;
  const u64 x = mulhi64(a << 9, TAG_LN2_Q64);                     // Q3.61
  const u64 den = (1ull << 63) - (mulhi64(E, E) << 1);            // Q1.63, in [3/4, 1)
  const u64 q = mulhi64(mulhi64(e, x), rcp_significand(den << 1));  // Q4.60, times 4 2^-k
  return 0 - (k <= 6 ? q << (6 - k) : q >> (k - 6));
}

// 1 - the Stolarsky mean's factor
//   2 (g - 1)/g (1 - 2^(-g D)) / ((1 - 2^(-(g - 1) D)) (1 + E))
// from g as Q2.61 and 2 (g - 1)/g as Q0.64 (1.3 <= g <= 1.9: exp2_fraction is good to 2^-58.7
// and 1 - 2^(1 - g) above 0.18).
TAG_HD u64 stolarsky_deficit_middle(u64 a, u64 g_q61, u64 fac_q64) {
  const u64 one = 1ull << 63, D = a << 7;                          // Q4.59
  const u64 gD = (mulhi64(D, g_q61) << 3) | ((D * g_q61) >> 61);   // Q4.59
  const u64 hD = mulhi64(a << 9, (g_q61 - (1ull << 61)) << 3);     // (g - 1) D, Q3.61
  const u64 num = one - exp2_negative<59>(gD);
  const u64 den = mulhi64(one - exp2_negative<61>(hD), one + exp2_negative<52>(a));  // Q2.62
  const int lz = leading_zeros(den);
  return 0 - (mulhi64(mulhi64(num, rcp_significand(den << lz)), fac_q64) << lz);
}

// 1 - c (Q0.64) for c of the middle range
TAG_HD double middle_factor(u64 c) {
  const u64 f = 0 - c;
  const int lz = leading_zeros(f);
  return f64_from(((u64)(1021 - lz) << 52) + round53(f << lz));
}

// The Stolarsky mean S(u, v) = (g-1)/g (v^g - u^g)/(v^(g-1) - u^(g-1)) is
// (u + v)/2 times sinh(g x) (g-1)/g / (sinh((g-1) x) cosh(x)), x = log(v/u)/2:
// the coefficients of that factor in z = d^2, x = d ln2/2, from the quotient of
// the three Taylor series.
inline EvenSeries stolarsky_series(double gamma) {
  constexpr int T = 14;
  using R = long double;
  const R g = gamma, ln2h = 0.346573590279972654708616060729088284L, x2 = ln2h * ln2h;
  R num[T], den[T], sb[T], ch[T];
  R p = 1, q = 1, r = 1;
  for (int k = 0; k < T; ++k) {  // sinh(gx)/(gx), sinh((g-1)x)/((g-1)x), cosh(x)
    num[k] = p;
    sb[k] = q;
    ch[k] = r;
    p *= g * g * x2 / ((2 * k + 2) * (R)(2 * k + 3));
    q *= (g - 1) * (g - 1) * x2 / ((2 * k + 2) * (R)(2 * k + 3));
    r *= x2 / ((2 * k + 1) * (R)(2 * k + 2));
  }
  R w[T];
  for (int k = 0; k < T; ++k) {
    den[k] = 0;
    for (int i = 0; i <= k; ++i) den[k] += sb[i] * ch[k - i];
  }
  for (int k = 0; k < T; ++k) {
    w[k] = num[k];
    for (int i = 1; i <= k; ++i) w[k] -= den[i] * w[k - i];
  }
  EvenSeries s{};
  s.ok = gamma > 1.0 && gamma < 2.0;
  R at1 = 0;
  for (int k = 0; k < 13; ++k) {
    const R a = -w[k + 1];
    at1 += a;
    if (k < 7)
      s.a[k] = (i64)llroundl(a * 9223372036854775808.0L);
    else
      s.b[k - 7] = (float)a;
    if (k == 0 && !(a >= 0 && a < 0.25L)) s.ok = 0;
    if (k == 7 && !(fabsl(a) < 1e-9L)) s.ok = 0;
  }
  if (!(at1 >= 0 && at1 < 0.25L)) s.ok = 0;
  return s;
}

}  // namespace tag
