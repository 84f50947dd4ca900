// Two-point fluxes in element-wide fixed point on the integer pipe.
//
// Why: the volume integral is nothing but products and sums of node values, and
// GB300 runs those faster as 64-bit integer words than on its FP64 pipe.  An
// FP64 operation occupies an SM for 20 cycles per warp (measured 1.57 per clock);
// the product hmul below takes 3.4, a sum 1.
//
// Words: m stands for m 2^(s - 64) with one exponent s per field and element,
// chosen from the element's largest values so that every intermediate stays in
// (-1/2, 1/2): |m| < 2^63 without a run-time test.  A node field below 1/4 of its
// scale keeps 62 bits relative to the element's largest value; a product rounds
// at 2^-64 of its scale, which the bounds of fx_scale place near the result.
//
// Weights: with the quadrature weights w, Q_ab = w_a Dsplit_ab is antisymmetric,
// so one product Q_ab n serves both nodes of a pair, the surface fluxes join the
// sums unweighted, and 1/w_a is applied once per node and direction.  Sums of
// words are exact and independent of their order.
//
// Measured on the shell at polydeg 5 (2,654,208 nodes): the element kernel 2.15
// ms in FP64 (its pipe 90 % busy) and 0.93 ms in words (issue slots 55 %, integer
// pipes 50 % busy); its error against extended precision is 0.4 to 0.8 of the
// FP64 form's.
//
// Elements whose values leave the scales' range (infinities, NaN, magnitudes
// beyond 2^+-150) take the FP64 form.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstring>

#include "tag_common.cuh"

namespace tag {

// a b / 2^64 (error within +-2, 0.5 rms).  Only unsigned 32-bit products are one
// instruction here (a signed widening one takes three), so the operands are
// offset by 2^63: a b = a' b' - 2^63 (a + b) - 2^126, where a' costs one
// exclusive or and a/2 a shift, both shared by the products of one operand.
// Measured in SM cycles per warp: 3.4, against 7.2 of three signed products
// and 7.2 of __mul64hi (an FP64 operation: 20).
// 0.75 low on average, which sums of products add once.
TAG_HD u64 offset_word(i64 a) { return (u64)a ^ 0x8000000000000000ull; }
constexpr u64 kOffset = 1ull << 62;  // 2^126 / 2^64
TAG_HD i64 hmul_raw(i64 a, i64 b) {
  return (i64)(umul_high(offset_word(a), offset_word(b)) - kOffset) - (a >> 1) - (b >> 1);
}
TAG_HD i64 hmul(i64 a, i64 b) { return hmul_raw(a, b) + 1; }
// for b >= 0 (1 low)
TAG_HD i64 hmul_pos(i64 a, i64 b) {
  return (i64)umul_high(offset_word(a), (u64)b) - (b >> 1) + 1;
}

// x < 2^e as a word of scale e + 2: x 2^(62 - e), towards zero.
TAG_HD i64 to_fixed(double x, int e) {
  const u64 b = f64_bits(x);
  const int E = (int)f64_exponent(b);
  const int sh = e + 1022 - E;
  u64 m = ((b & 0x000fffffffffffffull) | 0x0010000000000000ull) << 9;
  m = E == 0 || sh > 63 ? 0 : m >> sh;
  return (i64)b < 0 ? (i64)(0 - m) : (i64)m;
}

// m 2^(s - 64), rounded once (s within +-900).
TAG_HD double from_fixed(i64 m, int s) {
  if (m == 0) return 0.0;
  const u64 a = magnitude(m);
#ifdef __CUDA_ARCH__
  const int lz = __clzll((i64)a);
#else
  const int lz = __builtin_clzll(a);
#endif
  const u64 r = ((u64)(1021 + s - lz) << 52) + round53(a << lz);
  return f64_from(r | ((u64)m & 0x8000000000000000ull));
}

// Basis in words (FxBasis::ok: the operator is antisymmetric, as it is on
// Legendre-Gauss-Lobatto nodes): Q[a n + b] = w_a Dsplit_ab / 2 2^(64 - sq), each
// below 1/2 and a row's magnitudes summing to at most 1; W[a] = 2^(64 - kw) / w_a
// below 1/2.
struct FxBasis {
  i64 Q[64];
  i64 W[8];
  float one, row;  // the largest |Q_ab| and row sum, as fractions of 2^sq
  int S[2];        // relative change of the first and last node's weight, times 2^63
  int sq, kw, ok, pad;  // (a multiple of 16 bytes)
};

inline void load_fixed_basis(FxBasis& f, const double* Ds, const double* w, int n) {
  std::memset(&f, 0, sizeof(f));
  double row = 0.0, one = 0.0, skew = 0.0, winv = 0.0;
  for (int a = 0; a < n; ++a) {
    double s = 0.0;
    for (int b = 0; b < n; ++b) {
      if (b == a) continue;
      const double q = 0.5 * w[a] * Ds[a * n + b];
      s += std::fabs(q);
      one = std::fmax(one, std::fabs(q));
      skew = std::fmax(skew, std::fabs(q + 0.5 * w[b] * Ds[b * n + a]));
    }
    row = std::fmax(row, s);
    winv = std::fmax(winv, 1.0 / w[a]);
  }
  f.ok = row > 0.0 && skew <= 1e-12 * row && std::isfinite(row) && std::isfinite(winv);
  if (!f.ok) return;
  f.sq = std::max(std::ilogb(row) + 1, std::ilogb(one) + 2);
  f.kw = std::ilogb(winv) + 2;
  f.one = (float)std::ldexp(one, -f.sq) * 1.00001f;
  f.row = (float)std::ldexp(row, -f.sq) * 1.00001f;
  // The weights and the operator are rounded by themselves, so w_a Dsplit_ab and
  // -w_b Dsplit_ba differ in their last places: the weights are adjusted to the
  // least sum of those relative differences squared (by a few 1e-16), and the
  // mean of the two is taken, so that Q_ab / w_a is as near Dsplit_ab as one
  // antisymmetric matrix can be.  The surface fluxes, whose weight stays 1/w, are
  // scaled by the change (S).
  long double ww[8];
  for (int a = 0; a < n; ++a) {
    long double r = 0.0L;
    for (int b = 0; b < n; ++b)
      if (b != a && Ds[a * n + b] != 0.0)
        r += (long double)w[a] * Ds[a * n + b] / (-(long double)w[b] * Ds[b * n + a]) - 1.0L;
    ww[a] = w[a] * (1.0L - r / n);
  }
  for (int a = 0; a < n; ++a) {
    for (int b = 0; b < n; ++b) {
      if (b == a) continue;
      const long double q = 0.25L * (ww[a] * Ds[a * n + b] - ww[b] * Ds[b * n + a]);
      f.Q[a * n + b] = (i64)llroundl(ldexpl(q, 64 - f.sq));
    }
    f.W[a] = (i64)llroundl(ldexpl(1.0L / ww[a], 64 - f.kw));
  }
  f.S[0] = (int)lroundl(ldexpl(ww[0] / w[0] - 1.0L, 63));
  f.S[1] = (int)lroundl(ldexpl(ww[n - 1] / w[n - 1] - 1.0L, 63));
}

// Largest magnitudes of an element's fields, as high words of the doubles
// (their order is the values'), and the scales chosen from them.
// Velocities by component, so that sums of components and normal velocities are
// bounded by their own values: a place or two of every word.  (Shell elements
// 15 km tall, whose density falls by e^2, need it: without, their energy error at
// polydeg 7 was 1.35 of the FP64 form's, now 0.8.)
enum FxMax : int {
  kMxV = 0, kMxRho = kMxV + 3, kMxP, kMxX, kMxG, kMxN, kMxF = kMxN + 3, kMxCount = kMxF + 9
};

struct FxScale {
  int sv, sr, sp, sx, sg;  // velocities (halved), density, pressure, transported scalar's node
                           // value, geopotential differences
  int sh;                  // the scalar's flux over the normal velocity (rho x + p/2)
  int jh;                  // left shift of that sum
  int sn[3], kq[3];        // contravariant vectors per direction; left shift of Q n
  int ok;
};
constexpr int kFxDoubles = (sizeof(FxScale) + 7) / 8;  // its place in shared memory

TAG_HD u32 high_magnitude(double x) { return (u32)(f64_bits(x) >> 32) & 0x7fffffffu; }

// 2^k, and an upper bound of a high word's double over 2^s
TAG_HD float pow2f(int k) { return f32_from((u32)(127 + max(-100, min(k, 100))) << 23); }
TAG_HD float fx_fraction(u32 hi, int s) {
  const float m = f32_from(0x3f800000u + ((hi & 0xfffffu) << 3) + 8u);  // [1, 2]
  return m * pow2f((int)(hi >> 20) - 1023 - s);
}

// The largest k with x 2^k <= top (x > 0; 120 for x = 0), and a bound x of scale s
// brought under top by raising s.
TAG_HD int fx_room(float x, float top) {
  if (!(x > 1e-30f)) return x == x ? 120 : 0;
  // by the exponents of x and top, one less where x's significand is larger
  const u32 bx = f32_bits(x), bt = f32_bits(top);
  return (int)(bt >> 23) - (int)(bx >> 23) - ((bx & 0x7fffffu) > (bt & 0x7fffffu) ? 1 : 0);
}
TAG_HD void fx_fit(float& x, int& s, float top) {
  const int k = min(0, fx_room(x, top));
  x *= pow2f(k);
  s -= k;
}

// Scales of an element from its maxima mx (kMxF + 3 kind + d: surface fluxes of
// the mass, the momentum and the transported scalar on direction d's faces) in
// `dims` directions.  Each is the smallest that bounds the words derived from it
// by 1/2, the bounds being products of the maxima themselves.
TAG_HD FxScale fx_scale(const u32* mx, int dims, const FxBasis& b) {
  const float top = 0.48f;
  bool ok = b.ok != 0;
  int e[kMxCount];  // value < 2^e
  for (int k = 0; k < kMxCount; ++k) {
    const int x = (int)(mx[k] >> 20) - 1022;
    ok = ok && x <= 150;  // infinities and NaN have x = 1025
    e[k] = x < -150 ? -150 : x;
  }
  FxScale s;
  s.ok = ok ? 1 : 0;
  s.sr = e[kMxRho] + 2;
  s.sg = e[kMxG] + 2;
  int ev = -150;
  for (int c = 0; c < dims; ++c) ev = max(ev, e[kMxV + c]);
  // so that the sums of a node's components and of two nodes' values fit a word
  s.sv = ev + 2;
  float sum = 0.0f, most_v = 0.0f;
  for (int c = 0; c < dims; ++c) {
    const float f = fx_fraction(mx[kMxV + c], s.sv);
    sum += f;
    most_v = fmaxf(most_v, f);
  }
  if (!(fmaxf(sum, 2.0f * most_v) <= 0.49f)) s.sv = ev + 3;
  for (int d = 0; d < 3; ++d) {
    s.sn[d] = d < dims ? e[kMxN + d] + 3 : 0;
    s.kq[d] = 0;
  }
  for (int d = 0; d < dims; ++d)  // surface mass fluxes to 1/16
    s.sv = max(s.sv, e[kMxF + d] + 4 - s.sr - s.sn[d] - b.sq);
  const float rho = 2.0f * fx_fraction(mx[kMxRho], s.sr),
              g = 2.0f * fx_fraction(mx[kMxG], s.sg);
  float v = 0.0f, v1 = 0.0f, vv = 0.0f;  // largest component, their sum, sum of squares
  for (int c = 0; c < dims; ++c) {
    const float f = fx_fraction(mx[kMxV + c], s.sv);
    v = fmaxf(v, f);
    v1 += f;
    vv += f * f;
  }
  // x = mean(scalar) + v.v
  s.sx = max(e[kMxX] + 2, 2 * s.sv);
  float x = 2.0f * fx_fraction(mx[kMxX], s.sx) + vv * pow2f(2 * s.sv - s.sx);
  fx_fit(x, s.sx, top);
  // pressure sum +- 2 rho_mean g
  s.sp = max(max(e[kMxP] + 2, s.sr + s.sg + 1), s.sr + 2 * s.sv);
  for (int d = 0; d < dims; ++d) s.sp = max(s.sp, e[kMxF + 3 + d] + 4 - s.sn[d] - b.sq);
  float pp = 2.0f * fx_fraction(mx[kMxP], s.sp) + rho * g * pow2f(s.sr + s.sg + 1 - s.sp);
  fx_fit(pp, s.sp, top);
  const float p = fx_fraction(mx[kMxP], s.sp);
  // h = rho_mean x + (p +- 2 rho_mean g) / 2, shifted left by jh
  s.sh = max(s.sr + s.sx, s.sp - 1);
  int fluxes = -10000;  // surface fluxes to 1/16
  for (int d = 0; d < dims; ++d)
    fluxes = max(fluxes, e[kMxF + 6 + d] + 3 - s.sv - s.sn[d] - b.sq);
  s.sh = max(s.sh, fluxes);
  float h = rho * x * pow2f(s.sr + s.sx - s.sh) + pp * pow2f(s.sp - 1 - s.sh);
  fx_fit(h, s.sh, top);
  s.jh = max(0, min(min(fx_room(h, top), s.sh - fluxes), 8));
  h *= pow2f(s.jh);
  s.sh -= s.jh;
  for (int d = 0; d < dims; ++d) {
    const float n = 2.0f * fx_fraction(mx[kMxN + d], s.sn[d]);
    const float vn = 2.0f * v1 * n;  // per unit of Q
    const float mass = rho * vn;
    const int sd = s.sn[d] + b.sq;
    float most = b.one * vn;
    most = fmaxf(most, b.row * mass + fx_fraction(mx[kMxF + d], s.sr + s.sv + sd));
    most = fmaxf(most, b.row * (n * pp + 2.0f * mass * v * pow2f(s.sr + 2 * s.sv - s.sp)) +
                           fx_fraction(mx[kMxF + 3 + d], s.sp + sd));
    most = fmaxf(most, b.row * vn * (h + p * pow2f(s.sp - 1 - s.sh)) +
                           0.5f * fx_fraction(mx[kMxF + 6 + d], s.sh + s.sv + sd));
    most = fmaxf(most, b.one * n);
    s.kq[d] = max(0, min(fx_room(most, top), 12));
    most *= pow2f(s.kq[d]);
    if (!(most <= 0.49f)) s.ok = 0;
  }
  return s;
}

// Scale of the sums of kind 0 mass, 1 momentum, 2 transported scalar in
// direction d (without the basis' part).
TAG_HD int fx_kind_scale(const FxScale& s, int kind) {
  return kind == 0 ? s.sr + s.sv : kind == 1 ? s.sp : s.sh + s.sv;
}
TAG_HD int fx_direction_scale(const FxScale& s, int d) { return s.sn[d] - s.kq[d]; }

// Shifts that bring a pair's terms to their sums' scales, taken of an operand
// before the product (which rounds; a shift of the product would truncate).
struct FxShift {
  int t, h, v, x, p, j;  // f v, 2 rho_mean g, v.v, rho_mean x and p/2 in h, h itself (left)
};
TAG_HD FxShift fx_shift(const FxScale& s) {
  FxShift k;
  k.t = min(s.sp - s.sr - 2 * s.sv, 63);
  k.h = min(s.sp - s.sr - s.sg - 1, 63);
  k.v = min(s.sx - 2 * s.sv, 63);
  k.x = min(s.sh + s.jh - s.sr - s.sx, 63);
  k.p = min(s.sh + s.jh - s.sp + 1, 63);
  k.j = s.jh;
  return k;
}

// The sum over the D directions of A[d stride] W_d (words of scales sd[d] + one
// common part, W_d >= 0), as a word whose scale is the common part + `scale`.
// The sums are cancelled ones: they are brought to the coarsest direction's
// scale and then up to the word's top before the products.
template <int D>
TAG_DEV i64 fx_weighted_sum(const i64* A, int stride, const i64* W, const int* node, const int* sd,
                            int& scale) {
  int top = sd[0];
#pragma unroll
  for (int d = 1; d < D; ++d) top = max(top, sd[d]);
  i64 a[D];
  u64 all = 0;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    a[d] = A[d * stride] >> min(top - sd[d], 63);
    all |= (u64)(a[d] ^ (a[d] >> 63));
  }
  // three leading zeros: three terms below 1/8 (a sum may need two places down)
  const int lz = __clzll((i64)all), up = max(lz - 3, 0), down = max(3 - lz, 0);
  i64 tot = 0;
#pragma unroll
  for (int d = 0; d < D; ++d) tot += hmul_pos((a[d] >> down) << up, W[node[d]]);
  scale = top - up + down;
  return tot;
}

// c with factor = 1 - c (Q0.64) of a logarithmic mean of two words of one scale
// from the difference of the logarithms; beyond a factor of 256 the far branch
// divides in FP64.
static __device__ __noinline__ u64 fx_far_deficit(i64 a, i64 b, i64 d, int inverse) {
  const u64 m = magnitude(d);
  if (middle_range(m))
    return inverse ? inv_ln_mean_deficit_middle(m) : ln_mean_deficit_middle(m);
  const double x = (double)a, y = (double)b;
  const double f = inverse ? inv_ln_factor_far(x, y, d) : ln_factor_far(x, y, d);
  return f < 1.0 && f > 0.0 ? (u64)((1.0 - f) * 18446744073709551616.0) : 0;
}
// The two means of a pair, each c by the form that fits its own difference.
TAG_DEV u64 fx_ln_deficit(i64 a, i64 b, i64 d) {
  const u64 m = magnitude(d);
  if (!series_in_range(m)) return fx_far_deficit(a, b, d, 0);
  const u64 z = log_square(m);
  return z < kShortZ ? ln_mean_deficit_short(z) : ln_mean_deficit(z);
}
TAG_DEV u64 fx_inv_ln_deficit(i64 a, i64 b, i64 d) {
  const u64 m = magnitude(d);
  if (!series_in_range(m)) return fx_far_deficit(a, b, d, 1);
  const u64 z = log_square(m);
  return z < kShortZ ? inv_ln_mean_deficit_short(z) : inv_ln_mean_deficit(z);
}
// s (1 - c) of a positive sum
TAG_DEV i64 fx_reduce(i64 s, u64 c) { return s - (i64)umul_high((u64)s, c) - 1; }

// Node values of one element's words: rho/2, the halved velocities, p/2, the
// geopotential's quarter relative to the element's first node, the transported
// scalar's node value, then two logarithm words that are kept.  The velocities
// are stored with their offset (a sum of two offset words is the plain sum).
template <int D>
TAG_DEV void fx_convert_node(double* q, const FxScale& s) {
  i64* w = reinterpret_cast<i64*>(q);
  w[0] = to_fixed(q[0], s.sr - 2);
#pragma unroll
  for (int k = 1; k <= D; ++k) w[k] = (i64)offset_word(to_fixed(q[k], s.sv - 2));
  w[D + 1] = to_fixed(q[D + 1], s.sp - 2);
  w[D + 2] = to_fixed(q[D + 2], s.sg - 2);
  w[D + 3] = to_fixed(q[D + 3], s.sx - 2);
}

// The pair flux of the energy equations (volume_pair of PhysEnergy2D / 3D) in
// words, weighted by Q_ab >= 0 (the caller orders the pair so): node a adds Fa,
// node b subtracts Fb.  The scalar's
// flux is regrouped as
//   vn (rho_mean x + (p +- 2 rho_mean g) / 2) + (p_a - p_b)(vn_b - vn_a) / 2,
// whose factor of vn is one word near its top.  27 (3D) or 20 (2D) products.
template <int D>
TAG_DEV void fx_energy_pair(const i64* qa, const i64* qb, const i64* na, const i64* nb, i64 Q,
                            const FxShift& k, int kq, i64* Fa, i64* Fb) {
  const i64 rho = fx_reduce(qa[0] + qb[0], fx_ln_deficit(qa[0], qb[0], qb[D + 4] - qa[D + 4]));
  i64 x = fx_reduce(qa[D + 3] + qb[D + 3],
                    fx_inv_ln_deficit(qa[D + 3], qb[D + 3], qb[D + 5] - qa[D + 5]));
  // normal velocities of both nodes and v_a.v_b: each product's offset terms
  // are collected, halves of the components' sums for the velocities
  i64 nq[D], hq = 0;
  u64 ua = 0, ub = 0;
  u64 va = 0, vb = 0, vv = 0;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    nq[d] = hmul_pos(na[d] + nb[d], Q) << kq;
    const u64 nw = offset_word(nq[d]), wa = (u64)qa[1 + d], wb = (u64)qb[1 + d];
    va += umul_high(nw, wa);
    vb += umul_high(nw, wb);
    vv += umul_high(wa, wb);
    hq += nq[d] >> 1;
    ua += offset_word(qa[1 + d]);
    ub += offset_word(qb[1 + d]);
  }
  const i64 sa = (i64)ua >> 1, sb = (i64)ub >> 1;
  constexpr u64 kDot = D * kOffset - D;  // modulo 2^64; the sums themselves fit
  const i64 vna = (i64)(va - kDot - (u64)(hq + sa)), vnb = (i64)(vb - kDot - (u64)(hq + sb));
  x += (i64)(vv - kDot - (u64)(sa + sb)) >> k.v;
  const i64 vn = vna + vnb, f1 = hmul_pos(vn, rho);
  const i64 h = hmul_pos((qb[D + 2] - qa[D + 2]) >> k.h, rho), p = qa[D + 1] + qb[D + 1];
  const i64 pp = p + h, pm = p - h;
  const u64 wp = offset_word(pp), wm = offset_word(pm);
  const i64 fs = f1 >> k.t;
  const u64 c = (u64)(fs >> 1) + 2 * kOffset - 2;
  const u64 cp = c + (u64)(pp >> 1), cm = c + (u64)(pm >> 1) + 1;
  const u64 wf = offset_word(fs);
  Fa[0] = f1;
  Fb[0] = f1;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const i64 v = (i64)((u64)qa[1 + d] + (u64)qb[1 + d]);
    const u64 t = umul_high(wf, offset_word(v)) - (u64)((v >> 1) + (nq[d] >> 1));
    const u64 nw = offset_word(nq[d]);
    Fa[1 + d] = (i64)(t + umul_high(nw, wp) - cp);
    Fb[1 + d] = (i64)(t + umul_high(nw, wm) - cm);
  }
  const i64 rx = hmul_pos(x, rho) >> k.x;
  const i64 w = hmul_raw(((qa[D + 1] - qb[D + 1]) >> k.p) << k.j, vnb - vna);
  Fa[D + 1] = hmul_raw(vn, (rx + (pp >> k.p)) << k.j) + w + 2;
  Fb[D + 1] = hmul_raw(vn, (rx + (pm >> k.p)) << k.j) + w + 1;
}

// A surface flux below half of its sum's scale 2^s as a word of that scale, with
// the end weight's change.
TAG_HD i64 fx_surface(double f, int s, int change) {
  const i64 m = to_fixed(f, s - 1) << 1;
  return m + (((i64)(int)(m >> 32) * change) >> 31);
}

// Maximum over a warp into a shared word.
TAG_DEV void warp_max_into(u32* dst, u32 v) {
  const u32 m = __reduce_max_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0 && m) atomicMax(dst, m);
}

}  // namespace tag
