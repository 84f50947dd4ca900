// Two-point fluxes in element-wide fixed point on the integer pipe.
//
// Why: the volume integral is nothing but products and sums of node values, and
// GB300 runs those faster as 64-bit integer words than on its FP64 pipe.  An
// FP64 operation occupies an SM for 20 cycles per warp (measured 1.57 per clock);
// the product hmul below takes 3.4, a sum 1.
//
// Words: m stands for m 2^(s - 64) with one exponent s per field, component and
// element, chosen from the element's largest values so that every intermediate
// stays in (-1/2, 1/2): |m| < 2^63 without a run-time test.  A node field below 1/4
// of its scale keeps 62 bits relative to the element's largest value; a product
// rounds at 2^-64 of its scale, which the bounds of fx_scale place near the result.
//
// Weights: with the quadrature weights w, Q_ab = w_a Dsplit_ab is antisymmetric,
// so one product Q_ab n serves both nodes of a pair, the surface fluxes join the
// sums unweighted, and 1/w_a is applied once per node and direction.  Sums of
// words are exact and independent of their order.
//
// Measured on the shell at polydeg 5 (2,654,208 nodes): right-hand side 2.32 ms
// with the FP64 form (its pipe 90 % busy), 1.11 ms in words.  Of that 0.04 ms are the
// scales by component.  With one scale per direction the horizontal momentum of
// flat elements lost up to eight places: its error against extended precision, over
// the FP64 form's, was 3 in elements 170 times as wide as tall and 320 at 20,000;
// it is 0.6 to 1.1 now at every width.
//
// Elements whose values leave the scales' range (infinities, NaN, magnitudes
// beyond 2^+-150) or spread too far (kMaxSpread) take the FP64 form.
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
// for b >= 0, with all 64 places for b (1 low)
TAG_HD i64 hmul_pos(i64 a, u64 b) { return (i64)(umul_high(offset_word(a), b) - (b >> 1)) + 1; }

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
  const int lz = leading_zeros(a);
  const u64 r = ((u64)(1021 + s - lz) << 52) + round53(a << lz);
  return f64_from(r | ((u64)m & 0x8000000000000000ull));
}

// Basis in words (FxBasis::ok: the operator is antisymmetric, as it is on
// Legendre-Gauss-Lobatto nodes): Q[a n + b] = |w_a Dsplit_ab| / 2 2^(64 - sq), each
// below 1, with the sign in the last place (1: negative); W[a] = 2^(64 - kw) / w_a
// below 1/2.
struct FxBasis {
  u64 Q[64];
  i64 W[8];
  float row;  // the largest row sum of |Q|, over 2^sq
  // the density's and the pressures' sums that leave a row room: mass fluxes to 0.36 for
  // normal velocities of 2 kTopV kTopN per unit of Q, pressure fluxes to 0.24
  float top_rho, top_p;
  int S[2];  // relative change of the first and last node's weight, times 2^63
  int sq, kw, ok;  // (a multiple of 16 bytes)
};
static_assert(sizeof(FxBasis) % 16 == 0, "16-byte aligned");

constexpr float kTop = 0.48f;   // bound of a word
constexpr float kTopV = 0.48f;  // of the sum of a node's velocity components
constexpr float kTopN = 0.49f;  // of two nodes' contravariant vectors

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
  f.sq = std::ilogb(one) + 1;
  f.kw = std::ilogb(winv) + 2;
  f.row = (float)std::ldexp(row, -f.sq) * 1.00001f;
  f.top_rho = std::fmin(kTop, 0.36f / (2.0f * kTopV * kTopN * f.row));
  f.top_p = std::fmin(kTop, 0.24f / (kTopN * f.row));
  // The weights and the operator are rounded by themselves, so w_a Dsplit_ab and
  // -w_b Dsplit_ba differ in their last places: the weights are adjusted to the
  // least sum of those relative differences squared (by a few 1e-16), and the
  // mean of the two is taken, so that Q_ab / w_a is as near Dsplit_ab as one
  // antisymmetric matrix can be.  The surface fluxes, whose weight stays the
  // rounded 1/w of the FP64 form (the end weights are 2 / (n (n - 1)): the quotient is
  // the exact integer, which the rounded weight's own inverse is not), are scaled by
  // the change (S).
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
      f.Q[a * n + b] = (u64)llroundl(ldexpl(fabsl(q), 63 - f.sq)) << 1 | (q < 0 ? 1 : 0);
    }
    f.W[a] = (i64)llroundl(ldexpl(1.0L / ww[a], 64 - f.kw));
  }
  f.S[0] = (int)lroundl(ldexpl(ww[0] * (1.0 / w[0]) - 1.0L, 63));
  f.S[1] = (int)lroundl(ldexpl(ww[n - 1] * (1.0 / w[n - 1]) - 1.0L, 63));
}

// Largest magnitudes of an element's fields, as high words of the doubles
// (their order is the values'), and the scales chosen from them.  Velocities,
// contravariant vectors and the surface fluxes of momentum by component: the
// vertical face of a flat element can be thousands of times its lateral ones,
// and a component that is small or zero must not be rounded at the largest one's
// scale (kMxN, kMxFv: 3 group + component).  kMx...Low: the smallest density,
// pressure and transported scalar, as the largest of kHighInf less the high word.
// Groups of directions share their scales: in 3D each direction is one, in 2D both
// are (64-member ensemble run 6.78 -> 6.4 ms with the same errors; in 3D the lateral
// directions' roundings at the vertical one's scale made the energy error of tall
// shell elements 1.6 instead of 0.7 of the FP64 form's).
constexpr u32 kHighInf = 0x7ff00000u;
enum FxMax : int {
  kMxV = 0, kMxRho = kMxV + 3, kMxP, kMxX, kMxRhoLow, kMxPLow, kMxXLow, kMxG, kMxN,
  kMxFm = kMxN + 9, kMxFv = kMxFm + 3, kMxFe = kMxFv + 9, kMxCount = kMxFe + 3
};
TAG_HD constexpr int fx_groups(int dims) { return dims == 3 ? 3 : 1; }
TAG_HD constexpr int fx_group(int dims, int d) { return dims == 3 ? d : 0; }
// (in a system of `dims` directions)
TAG_HD constexpr bool fx_used(int k, int dims) {
  if (k < kMxRho) return k < dims;
  if (k < kMxN) return true;
  if (k < kMxFm || (k >= kMxFv && k < kMxFe)) {
    const int r = k - (k < kMxFm ? kMxN : kMxFv);
    return r / 3 < fx_groups(dims) && r % 3 < dims;
  }
  return k - (k < kMxFv ? kMxFm : kMxFe) < fx_groups(dims);
}

// Shifts that bring a pair's terms to their sums' scales, four to a word (a pair
// reads them all, and registers bound the warps in flight): of the weighted normal
// for the normal velocity and of the transported momentum for the momentum's sum,
// both by component (right); of v.v by component; of 2 rho_mean g, of rho_mean x
// and p/2 in h (right), of h itself (left).
struct alignas(16) FxShift {
  u32 n, t, v, hxpj;
};
TAG_HD int fx_byte(u32 w, int k) {
#ifdef __CUDA_ARCH__
  return (int)__byte_perm(w, 0u, 0x4440u + k);
#else
  return (int)(w >> (8 * k)) & 255;
#endif
}
template <int D>
struct alignas(16) FxScale {
  static constexpr int G = fx_groups(D);
  FxShift k[G];          // by group of directions
  int sn[G][3];          // scales: contravariant vectors by group and component,
  int sum[G][5];         // each variable's sums by group,
  int sv[3];             // velocities (halved),
  int sr, sp, sx, sg;    // density, pressure, transported scalar's node value, geopotential
  int ok;
  int zero[2], pad[2];   // at rest: the sums of mass and of the transported scalar are 0
};
// Whether variable v's sums are exactly 0 (their words are products of roundings).
template <int D>
TAG_HD bool fx_zero(const FxScale<D>& s, int v) {
  return (v == 0 && s.zero[0]) || (v == D + 1 && s.zero[1]);
}
template <int D>
constexpr int kFxDoubles = sizeof(FxScale<D>) / 8;  // its place in shared memory
static_assert(kFxDoubles<2> % 2 == 0 && kFxDoubles<3> % 2 == 0, "16-byte aligned");

TAG_HD u32 high_magnitude(double x) { return (u32)(f64_bits(x) >> 32) & 0x7fffffffu; }

// A node's values and contravariant vectors into the maxima by up(FxMax, magnitude).
// The words' products take densities as positive: bad states leave.
template <int D, class Up>
TAG_HD void fx_node_maxima(const double* q, const double* ja, Up up) {
#pragma unroll
  for (int c = 0; c < D; ++c) up(kMxV + c, high_magnitude(q[1 + c]));
  const u32 rho = not_positive(q[0]) ? kHighInf : high_magnitude(q[0]);
  const u32 p = not_positive(q[D + 1]) ? kHighInf : high_magnitude(q[D + 1]);
  const u32 x = not_positive(q[D + 3]) ? kHighInf : high_magnitude(q[D + 3]);
  up(kMxRho, rho);
  up(kMxP, p);
  up(kMxX, x);
  up(kMxRhoLow, kHighInf - rho);
  up(kMxPLow, kHighInf - p);
  up(kMxXLow, kHighInf - x);
  up(kMxG, high_magnitude(q[D + 2]));
#pragma unroll
  for (int k = 0; k < D * D; ++k)
    up(kMxN + 3 * fx_group(D, k / D) + k % D, high_magnitude(ja[k]));
}
// Place of the surface flux of variable v on direction d's faces.
template <int D>
TAG_HD constexpr int fx_face_max(int v, int d) {
  return v == 0 ? kMxFm + fx_group(D, d)
                : v == D + 1 ? kMxFe + fx_group(D, d) : kMxFv + 3 * fx_group(D, d) + v - 1;
}

// 2^k, and an upper bound of a high word's double over 2^s
TAG_HD float pow2f(int k) { return f32_from((u32)(127 + max(-100, min(k, 100))) << 23); }
TAG_HD float fx_fraction(u32 hi, int s) {
  const float m = f32_from(0x3f800000u + ((hi & 0xfffffu) << 3) + 8u);  // [1, 2]
  return m * pow2f((int)(hi >> 20) - 1023 - s);
}

// Half octaves that density, pressure or temperature may spread over within an
// element.  The words are rounded at the scale of an element's largest values, FP64
// numbers at their own, so the least dense nodes lose what the spread takes.  Error of
// the thinnest row of nodes against extended precision, over the FP64 form's, in an
// isothermal atmosphere at polydegs 3 and 5: up to 1.04 at 2^3 (15 km in one element),
// 1.6 at 2^4, 2.6 at 2^5, 6 at 2^6, 26 at 2^8; of the whole element 0.6 to 1.06 at
// every spread.
constexpr u32 kMaxSpread = 7;

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

// Scales of an element of D directions from its maxima: each is the smallest that
// bounds the words derived from it by 1/2, the bounds being products of the maxima
// themselves.  One call per group d of directions (the calls share no results, so that
// a thread each can take them); d = 0 also fills the common part.
//
// The weighted normals and the normal velocities of single pairs take the whole
// word: they are what cancels where the wind blows along an element's faces.  The
// room for the sums over a row of Q is left in density, pressure and h.
template <int D>
TAG_HD void fx_scale(const u32* mx, const FxBasis& b, int d, FxScale<D>& s) {
  // value < 2^e
  const auto e = [mx](int k) { return max((int)(mx[k] >> 20) - 1022, -150); };
  // velocities: the sums of a node's components and of two nodes' values fit a word
  int sv[D], most_v = -1000;
  float v[D], sum_v = 0.0f;
  u32 mass = 0, scalar = 0;
#pragma unroll
  for (int c = 0; c < D; ++c) {
    const u32 m = mx[kMxV + c];
    sv[c] = max((int)(m >> 20) - 1022, -150) + 2;
    v[c] = fx_fraction(m, sv[c]);
    sum_v += v[c];
    mass |= m | (c < fx_groups(D) ? mx[kMxFm + c] : 0u);
    scalar |= m | (c < fx_groups(D) ? mx[kMxFe + c] : 0u);
  }
#pragma unroll
  for (int c = 0; c < D; ++c) {
    if (!(sum_v <= kTopV)) {
      v[c] *= 0.5f;
      sum_v -= v[c];
      sv[c] += 1;
    }
    most_v = max(most_v, sv[c]);
  }
  // density sum
  int sr = e(kMxRho) + 2;
  float rho = 2.0f * fx_fraction(mx[kMxRho], sr);
  fx_fit(rho, sr, b.top_rho);
  // x = mean(scalar) + v.v
  int sx = max(e(kMxX) + 2, 2 * most_v);
  float x = 2.0f * fx_fraction(mx[kMxX], sx);
#pragma unroll
  for (int c = 0; c < D; ++c) x += v[c] * v[c] * pow2f(2 * sv[c] - sx);
  fx_fit(x, sx, kTop);
  // pressure sum +- 2 rho_mean g; a row's transported momentum to 0.1
  const int sg = e(kMxG) + 2;
  int sp = max(max(e(kMxP) + 2, sr + sg + 1), sr + 2 * most_v + 1);
  float pp = 2.0f * fx_fraction(mx[kMxP], sp) +
             rho * (2.0f * fx_fraction(mx[kMxG], sg)) * pow2f(sr + sg + 1 - sp);
  fx_fit(pp, sp, b.top_p);
  // This group's weighted normals Q n: scale sN by component; surface fluxes to 1/8.
  // The normal velocity: scale svn; vn: of a pair per unit of Q.
  int sN[D], svn = e(kMxFm + d) + 3 - sr;
  float vn = 0.0f;
#pragma unroll
  for (int c = 0; c < D; ++c) {
    const u32 m = mx[kMxN + 3 * d + c];
    sN[c] = max((int)(m >> 20) - 1022, -150) + 2;
    if (!(2.0f * fx_fraction(m, sN[c]) <= kTopN)) sN[c] += 1;
    sN[c] = max(sN[c] + b.sq, e(kMxFv + 3 * d + c) + 3 - sp);
    svn = max(svn, sN[c] + sv[c]);
  }
#pragma unroll
  for (int c = 0; c < D; ++c)
    vn += 4.0f * v[c] * fx_fraction(mx[kMxN + 3 * d + c], svn - sv[c] - b.sq);
  // h = rho_mean x + (p +- 2 rho_mean g) / 2, shifted left by kj: by what a row of it with
  // the pressures' difference and the surface fluxes leave
  int sh = max(sr + sx, sp - 1);
  const float h = rho * x * pow2f(sr + sx - sh) + pp * pow2f(sp - 1 - sh);
  const float row_h = b.row * vn * (h + fx_fraction(mx[kMxP], sp) * pow2f(sp - 1 - sh)) +
                      0.5f * fx_fraction(mx[kMxFe + d], sh + svn);
  const int room = min(fx_room(fmaxf(h, row_h), kTop), 8), kj = max(room, 0);
  sh -= room;
  FxShift k{};
#pragma unroll
  for (int c = 0; c < D; ++c) {
    sN[c] = max(sN[c], sr + svn + sv[c] - sp);
    k.n |= (u32)min(svn - sv[c] - sN[c], 63) << (8 * c);
    k.t |= (u32)min(sN[c] + sp - sr - svn - sv[c], 63) << (8 * c);
    k.v |= (u32)min(sx - 2 * sv[c], 63) << (8 * c);
    s.sn[d][c] = sN[c] - b.sq;
    s.sum[d][1 + c] = sN[c] + sp;
  }
  k.hxpj = (u32)min(sp - sr - sg - 1, 63) | (u32)min(sh + kj - sr - sx, 63) << 8 |
           (u32)min(sh + kj - sp + 1, 63) << 16 | (u32)kj << 24;
  s.k[d] = k;
  s.sum[d][0] = sr + svn;
  s.sum[d][D + 1] = sh + svn;
  if (d == 0) {
    u32 all = 0, spread = 0;
#pragma unroll
    for (int k = 0; k < kMxCount; ++k)
      if (fx_used(k, D)) all = max(all, mx[k]);
#pragma unroll
    for (int f = 0; f < 3; ++f)
      spread = max(spread, mx[kMxRho + f] + mx[kMxRhoLow + f] - kHighInf);
    // (infinities and NaN have the exponent 1025; high words order like logarithms; the
    // Low entries of values above 2^-150 are in the range, too)
    s.ok = b.ok != 0 && (int)(all >> 20) - 1022 <= 150 && spread <= kMaxSpread << 19;
#pragma unroll
    for (int c = 0; c < D; ++c) s.sv[c] = sv[c];
    s.sr = sr;
    s.sp = sp;
    s.sx = sx;
    s.sg = sg;
    s.zero[0] = mass == 0;
    s.zero[1] = scalar == 0;
  }
}

// The sum over the D directions of A[d stride] W_d (words of scales sd[d], W_d >=
// 0), as a word of scale `scale`.
// The sums are cancelled ones: they are brought to the coarsest direction's
// scale and then up to the word's top before the products.
template <int D>
TAG_HD i64 fx_weighted_sum(const i64* A, int stride, const i64* W, const int* node, const int* sd,
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
  const int lz = leading_zeros(all), up = max(lz - 3, 0), down = max(3 - lz, 0);
  i64 tot = 0;
#pragma unroll
  for (int d = 0; d < D; ++d) tot += hmul_pos((a[d] >> down) << up, W[node[d]]);
  scale = top - up + down;
  return tot;
}

// c with factor = 1 - c (Q0.64) of a logarithmic mean of two words of one scale
// from the difference of the logarithms; beyond a factor of 256 the far branch
// divides in FP64.
TAG_SLOW u64 fx_far_deficit(i64 a, i64 b, i64 d, int inverse) {
  const u64 m = magnitude(d);
  if (middle_range(m))
    return inverse ? inv_ln_mean_deficit_middle(m) : ln_mean_deficit_middle(m);
  const double x = (double)a, y = (double)b;
  const double f = inverse ? inv_ln_factor_far(x, y, d) : ln_factor_far(x, y, d);
  return f < 1.0 && f > 0.0 ? (u64)((1.0 - f) * 18446744073709551616.0) : 0;
}
// The two means of a pair, each c by the form that fits its own difference.
TAG_HD u64 fx_ln_deficit(i64 a, i64 b, i64 d) {
  const u64 m = magnitude(d);
  if (!series_in_range(m)) return fx_far_deficit(a, b, d, 0);
  const u64 z = log_square(m);
  return z < kShortZ ? ln_mean_deficit_short(z) : ln_mean_deficit(z);
}
TAG_HD u64 fx_inv_ln_deficit(i64 a, i64 b, i64 d) {
  const u64 m = magnitude(d);
  if (!series_in_range(m)) return fx_far_deficit(a, b, d, 1);
  const u64 z = log_square(m);
  return z < kShortZ ? inv_ln_mean_deficit_short(z) : inv_ln_mean_deficit(z);
}
// s (1 - c) of a positive sum
TAG_HD i64 fx_reduce(i64 s, u64 c) { return s - (i64)umul_high((u64)s, c) - 1; }

// Node values of one element's words: rho/2, the halved velocities, p/2, the
// geopotential's quarter relative to the element's first node, the transported
// scalar's node value, then two logarithm words that are kept.  The velocities
// are stored with their offset (a sum of two offset words is the plain sum).
template <int D>
TAG_HD void fx_convert_node(double* q, const FxScale<D>& s) {
  i64* w = reinterpret_cast<i64*>(q);
  w[0] = to_fixed(q[0], s.sr - 2);
#pragma unroll
  for (int c = 0; c < D; ++c) w[1 + c] = (i64)offset_word(to_fixed(q[1 + c], s.sv[c] - 2));
  w[D + 1] = to_fixed(q[D + 1], s.sp - 2);
  w[D + 2] = to_fixed(q[D + 2], s.sg - 2);
  w[D + 3] = to_fixed(q[D + 3], s.sx - 2);
}

// The pair flux of the energy equations (volume_pair of PhysEnergy2D / 3D) in
// words, weighted by Q_ab > 0 (the caller orders the pair so): node a adds Fa,
// node b subtracts Fb.  The scalar's
// flux is regrouped as
//   vn (rho_mean x + (p +- 2 rho_mean g) / 2) + (p_a - p_b)(vn_b - vn_a) / 2,
// whose factor of vn is one word near its top.  27 (3D) or 20 (2D) products.
template <int D>
TAG_HD void fx_energy_pair(const i64* qa, const i64* qb, const i64* na, const i64* nb, u64 Q,
                           const FxShift& k, i64* Fa, i64* Fb) {
  const i64 rho = fx_reduce(qa[0] + qb[0], fx_ln_deficit(qa[0], qb[0], qb[D + 4] - qa[D + 4]));
  i64 x = fx_reduce(qa[D + 3] + qb[D + 3],
                    fx_inv_ln_deficit(qa[D + 3], qb[D + 3], qb[D + 5] - qa[D + 5]));
  // normal velocities of both nodes and v_a.v_b: each product's offset terms
  // are collected, halves of the components' sums for the velocities
  i64 nq[D], v[D], hq = 0;
  u64 ua = 0, ub = 0;
  u64 va = 0, vb = 0;
#pragma unroll
  for (int c = 0; c < D; ++c) {
    nq[c] = hmul_pos(na[c] + nb[c], Q);
    const i64 nv = nq[c] >> fx_byte(k.n, c);
    const u64 nw = offset_word(nv), wa = (u64)qa[1 + c], wb = (u64)qb[1 + c];
    va += umul_high(nw, wa);
    vb += umul_high(nw, wb);
    hq += nv >> 1;
    ua += offset_word(qa[1 + c]);
    ub += offset_word(qb[1 + c]);
    v[c] = (i64)(wa + wb);
    x += (i64)(umul_high(wa, wb) - (u64)(v[c] >> 1) - (kOffset - 1)) >> fx_byte(k.v, c);
  }
  const i64 sa = (i64)ua >> 1, sb = (i64)ub >> 1;
  constexpr u64 kDot = D * kOffset - D;  // modulo 2^64; the sums themselves fit
  const i64 vna = (i64)(va - kDot - (u64)(hq + sa)), vnb = (i64)(vb - kDot - (u64)(hq + sb));
  const i64 vn = vna + vnb, f1 = hmul_pos(vn, rho);
  const int kx = fx_byte(k.hxpj, 1), kp = fx_byte(k.hxpj, 2), kj = fx_byte(k.hxpj, 3);
  const i64 h = hmul_pos((qb[D + 2] - qa[D + 2]) >> fx_byte(k.hxpj, 0), rho), p = qa[D + 1] + qb[D + 1];
  const i64 pp = p + h, pm = p - h;
  const u64 wf = offset_word(f1), wp = offset_word(pp), wm = offset_word(pm);
  const u64 cf = kOffset - 1 + (u64)(f1 >> 1);
  const u64 cp = kOffset - 1 + (u64)(pp >> 1), cm = kOffset - 1 + (u64)(pm >> 1);
  Fa[0] = f1;
  Fb[0] = f1;
#pragma unroll
  for (int c = 0; c < D; ++c) {
    const i64 t = (i64)(umul_high(wf, offset_word(v[c])) - (u64)(v[c] >> 1) - cf) >> fx_byte(k.t, c);
    const u64 nw = offset_word(nq[c]), base = (u64)(t - (nq[c] >> 1));
    Fa[1 + c] = (i64)(base + umul_high(nw, wp) - cp);
    Fb[1 + c] = (i64)(base + umul_high(nw, wm) - cm);
  }
  const i64 rx = hmul_pos(x, rho) >> kx;
  const i64 w = hmul_raw(((qa[D + 1] - qb[D + 1]) >> kp) << kj, vnb - vna);
  Fa[D + 1] = hmul_raw(vn, (rx + (pp >> kp)) << kj) + w + 2;
  Fb[D + 1] = hmul_raw(vn, (rx + (pm >> kp)) << kj) + w + 1;
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
