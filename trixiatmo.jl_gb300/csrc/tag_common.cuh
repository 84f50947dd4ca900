// Shared device helpers for the DGSEM kernels (FP64 on CUDA cores).
#pragma once
#include <cstdint>
#include <string>
#include <cuda_runtime.h>

#include "../../include/trixiatmo_gpu.h"
#include "int_math.cuh"

#define TAG_DEV __device__ __forceinline__

namespace tag {

// Sets the message tag_last_error() returns on this thread (defined in tag_api.cu).
void set_last_error(const std::string& msg);

constexpr int kMaxNodes = 8;  // n = polydeg + 1 supported up to polydeg 7

// Factors of the logarithmic means of a node pair, from the difference d of
// their log2_fixed node logarithms (b minus a):
//   ln_mean(xa, xb) = (xa + xb)/2 R,  inv_ln_mean(1/ya, 1/yb) = (ya + yb)/2 Q.
// Values within a factor of two (every pair of an element that resolves its
// stratification) take the integer series, whatever their size: no reciprocal,
// no logarithm, no branch that splits a warp.  Up to a factor of 256 (vertical
// pairs of elements some 5 km tall and more, edges of clouds) an exponential of d
// and a reciprocal in words; beyond, d itself is the logarithm of the definition.
TAG_HD double log_of_difference(i64 d) { return (double)d * 1.539095918623324e-16; }  // ln2 2^-52

// Values of opposite sign, which partial densities and bad states may have, give
// NaN: the logarithm of their ratio.  Beside a zero the mean is 0 and its inverse
// has no value.
TAG_HD bool opposite_signs(double a, double b) { return (i64)(f64_bits(a) ^ f64_bits(b)) < 0; }
TAG_HD bool is_zero(double x) { return (f64_bits(x) << 1) == 0; }
TAG_HD double quiet_nan() { return f64_from(0x7ff8000000000000ull); }
// A node value whose inverse is averaged: NaN in place of zero.
TAG_HD double invertible(double x) { return is_zero(x) ? quiet_nan() : x; }
TAG_SLOW double ln_factor_far(double xa, double xb, i64 d) {
  if (opposite_signs(xa, xb)) return quiet_nan();
  if (is_zero(xa) || is_zero(xb)) return 0.0;
  const u64 a = magnitude(d);
  if (middle_range(a)) return middle_factor(ln_mean_deficit_middle(a));
  return int_div(2.0 * (xb - xa), log_of_difference(d) * (xa + xb));
}
TAG_SLOW double inv_ln_factor_far(double ya, double yb, i64 d) {
  if (opposite_signs(ya, yb) || is_zero(ya) || is_zero(yb)) return quiet_nan();
  const u64 a = magnitude(d);
  if (middle_range(a)) return middle_factor(inv_ln_mean_deficit_middle(a));
  return int_div(2.0 * ya * yb * log_of_difference(d), (yb - ya) * (ya + yb));
}
TAG_HD double ln_factor(double xa, double xb, i64 d) {
  const u64 a = magnitude(d);
  return series_in_range(a) ? ln_mean_factor(log_square(a)) : ln_factor_far(xa, xb, d);
}
TAG_HD double inv_ln_factor(double ya, double yb, i64 d) {
  const u64 a = magnitude(d);
  return series_in_range(a) ? inv_ln_mean_factor(log_square(a)) : inv_ln_factor_far(ya, yb, d);
}

// The means of two values themselves (interface kernels): ln_mean(x, y), and
// inv_ln_mean(1/x, 1/y) from the reciprocals' own values.
TAG_HD double ln_mean_of(double x, double y) {
  return 0.5 * (x + y) * ln_factor(x, y, log2_fixed(y) - log2_fixed(x));
}
TAG_HD double inv_ln_mean_of_reciprocals(double x, double y) {
  return 0.5 * (x + y) * inv_ln_factor(x, y, log2_fixed(y) - log2_fixed(x));
}

// Node logarithms are kept among the other node quantities as raw words.
TAG_HD double log_word(double x) { return f64_from((u64)log2_fixed(x)); }
// The same where values below zero are common: log2_fixed's words of negative
// values without its out-of-line branch.
TAG_HD double log_word_signed(double x) {
  const u64 b = f64_bits(x);
  return f64_from((u64)log2_fixed(f64_from(b & 0x7fffffffffffffffull)) + ((b >> 63) << 62));
}
TAG_HD i64 log_difference(double wa, double wb) { return (i64)(f64_bits(wb) - f64_bits(wa)); }

// FP64 forms of the two means, which the diagnostics (tag_means.cu) hold beside
// the kernels' integer forms.  With f2 = ((y-x)/(y+x))^2 and z = sqrt(f2):
//   ln_mean(x, y)     = (x+y)/2 * z/atanh(z) = (x+y)/2 * R(f2)
//   inv_ln_mean(x, y) = 2/(x+y) * atanh(z)/z = 2/(x+y) * Q(f2)
// Below kShortF2 the four-term Taylor forms are exact to < 2e-17 relative.  On
// the wider ranges [0, F] R and Q are Chebyshev economizations of their Taylor
// series (C. Lanczos, J. Math. Phys. 17 (1938) 123-199; coefficients made and
// checked by csrc/log_mean_series.py): six coefficients each for F = kSeriesF2
// (exact to < 5e-19 relative), nine (R) and ten (Q) for F = kLongF2 (< 4e-18).
constexpr double kShortF2 = 1.0e-4;
constexpr double kSeriesF2 = 1.0e-2;
constexpr double kLongF2 = 0.09;

TAG_DEV double ln_short_R(double f2) {
  return fma(f2, fma(f2, fma(f2, -44.0 / 945.0, -4.0 / 45.0), -1.0 / 3.0), 1.0);
}
TAG_DEV double ln_short_Q(double f2) {
  return fma(f2, fma(f2, fma(f2, 1.0 / 7.0, 1.0 / 5.0), 1.0 / 3.0), 1.0);
}

// R and Q on [0, kSeriesF2]
TAG_DEV double ln_series_R(double f2) {
  double r = -0.01719901874634888;
  r = fma(r, f2, -0.021792151641765893);
  r = fma(r, f2, -0.030194027707754922);
  r = fma(r, f2, -0.0465608465041037);
  r = fma(r, f2, -0.08888888888893755);
  r = fma(r, f2, -0.3333333333333333);
  return fma(r, f2, 1.0);
}
TAG_DEV double ln_series_Q(double f2) {
  double r = 0.07895661799581076;
  r = fma(r, f2, 0.09088609072099012);
  r = fma(r, f2, 0.11111123067087354);
  r = fma(r, f2, 0.14285714257655663);
  r = fma(r, f2, 0.20000000000024065);
  r = fma(r, f2, 0.3333333333333333);
  return fma(r, f2, 1.0);
}

// R and Q on [0, kLongF2]
TAG_DEV double ln_series_R_long(double f2) {
  double r = -0.013669329626825622;
  r = fma(r, f2, -0.01045355622562932);
  r = fma(r, f2, -0.013573328231670736);
  r = fma(r, f2, -0.016783737201999518);
  r = fma(r, f2, -0.02179692429315078);
  r = fma(r, f2, -0.030194001406289393);
  r = fma(r, f2, -0.04656084657952881);
  r = fma(r, f2, -0.08888888888882568);
  r = fma(r, f2, -0.33333333333333337);
  return fma(r, f2, 1.0);
}
TAG_DEV double ln_series_Q_long(double f2) {
  double r = 0.07283496074780077;
  r = fma(r, f2, 0.047418568133941144);
  r = fma(r, f2, 0.05939688448611953);
  r = fma(r, f2, 0.06662915697122629);
  r = fma(r, f2, 0.07692458351815545);
  r = fma(r, f2, 0.09090905424531916);
  r = fma(r, f2, 0.11111111162196165);
  r = fma(r, f2, 0.14285714285353665);
  r = fma(r, f2, 0.20000000000000986);
  r = fma(r, f2, 0.3333333333333333);
  return fma(r, f2, 1.0);
}

// Out-of-line branch of ln_mean_pair_halved for a pair with f2 at or above
// the series range lim (kLongF2 or kSeriesF2) in either mean, from the
// logarithms Lxa = log(xa/2) ... (differences do not see the halving).  One
// reciprocal serves both means: rho_mean = nx/ex and inv_beta_mean = ny/ey.
template <bool kLong>
static __device__ __noinline__ void ln_mean_pair_halved_log(double sx, double dx, double sy,
                                                            double dy, double f2x, double f2y,
                                                            double Lxa, double Lxb, double Lya,
                                                            double Lyb, double& rho_mean,
                                                            double& inv_beta_mean) {
  constexpr double lim = kLong ? kLongF2 : kSeriesF2;
  const bool lx = f2x >= lim, ly = f2y >= lim;
  const double Rx = kLong ? ln_series_R_long(f2x) : ln_series_R(f2x);
  const double Qy = kLong ? ln_series_Q_long(f2y) : ln_series_Q(f2y);
  const double nx = lx ? 2.0 * dx : sx * Rx;
  const double ny = ly ? Lyb - Lya : Qy;
  const double ex = lx ? Lxb - Lxa : 1.0;
  const double ey = ly ? 2.0 * dy : sy;
  const double r2 = 1.0 / (ex * ey);
  rho_mean = nx * ey * r2;
  inv_beta_mean = ny * ex * r2;
}

// ln_mean(x_a, x_b) and inv_ln_mean(y_a, y_b) from HALVED node values
// (hx = x/2, hy = y/2, which saves the factors 1/2 and 2 of the series forms:
// ln_mean = (hx_a + hx_b) R(f2x), inv_ln_mean = Q(f2y) / (hy_a + hy_b)), one
// reciprocal per pair.  Each mean takes the form its own f2 selects: the
// four-term series below kShortF2 (when kShort), else the polynomial on
// [0, kLongF2] (kLong) or [0, kSeriesF2]; logarithms for both once either f2
// is beyond that range.
template <bool kShort = true, bool kLong = true>
TAG_DEV void ln_mean_pair_halved(double hxa, double hxb, double hya, double hyb, double Lxa,
                                 double Lxb, double Lya, double Lyb, double& rho_mean,
                                 double& inv_beta_mean) {
  constexpr double lim = kLong ? kLongF2 : kSeriesF2;
  const double sx = hxa + hxb, dx = hxb - hxa;
  const double sy = hya + hyb, dy = hyb - hya;
  const double r = 1.0 / (sx * sy);
  const double isx = sy * r, isy = sx * r;
  const double tx = dx * isx, ty = dy * isy;
  const double f2x = tx * tx, f2y = ty * ty;
  const long long bx = __double_as_longlong(f2x), by = __double_as_longlong(f2y);
  if (max(bx, by) >= __double_as_longlong(lim)) {
    ln_mean_pair_halved_log<kLong>(sx, dx, sy, dy, f2x, f2y, Lxa, Lxb, Lya, Lyb,
                                                rho_mean, inv_beta_mean);
    return;
  }
  double R, Q;
  if (kShort && bx < __double_as_longlong(kShortF2))
    R = ln_short_R(f2x);
  else
    R = kLong ? ln_series_R_long(f2x) : ln_series_R(f2x);
  if (kShort && by < __double_as_longlong(kShortF2))
    Q = ln_short_Q(f2y);
  else
    Q = kLong ? ln_series_Q_long(f2y) : ln_series_Q(f2y);
  rho_mean = sx * R;
  inv_beta_mean = isy * Q;
}

// !(x > 0.0) and !isfinite(x) on the integer pipe (the FP64 pipe is the
// element kernels' bottleneck): IEEE bit patterns of positive doubles order
// like their values, and an exponent field of all ones is an infinity or NaN.
TAG_HD bool not_positive(double x) { return f64_bits(x) - 1ull >= 0x7ff0000000000000ull; }
TAG_HD bool not_finite(double x) {
  return (f64_bits(x) & 0x7ff0000000000000ull) == 0x7ff0000000000000ull;
}

// 2 x of a normal number with a normal double (an exponent increment on the
// integer pipe); zero becomes 2^-1022, which any product or sum absorbs.
TAG_HD double twice(double x) { return f64_from(f64_bits(x) + (1ull << 52)); }
// x / 2 of a normal number with a normal half
TAG_HD double half_of(double x) { return f64_from(f64_bits(x) - (1ull << 52)); }

// Programmatic dependent launch (launch_overlapped): a kernel lets the next one
// of its stream start once all its CTAs are past their main work (earlier, the
// next one's CTAs would fill the SMs unevenly), and that one loads what no kernel
// writes (geometry, indices, operators) before it waits for this one's end.  A launch without the attribute is unaffected.  What
// the previous kernels write is read after the wait, and through pointers
// without __restrict__, whose loads the compiler may not move across it.
TAG_DEV void release_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
TAG_DEV void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Face node (i, j) of face f (0 = xi-, 1 = xi+, 2 = eta-, 3 = eta+) at index l.
TAG_DEV void face_node(int f, int l, int n, int& i, int& j) {
  if (f < 2) {
    i = (f == 0) ? 0 : n - 1;
    j = l;
  } else {
    i = l;
    j = (f == 2) ? 0 : n - 1;
  }
}

// Block copies of `count` doubles by the threads of a CTA.  copy_in is
// asynchronous (wait with copy_in_wait before the barrier): 16 bytes per
// instruction where both sides allow it, 8 otherwise; no registers between.
TAG_DEV void copy_in(double* smem, const double* __restrict__ g, int count) {
  const u32 s = (u32)__cvta_generic_to_shared(smem);
  if (((((size_t)g) | s | (count * 8u)) & 15u) == 0) {
    for (int t = threadIdx.x; t < count / 2; t += blockDim.x)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s + 16 * t), "l"(g + 2 * t));
  } else {
    for (int t = threadIdx.x; t < count; t += blockDim.x)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s + 8 * t), "l"(g + t));
  }
}
// The same for `ne` blocks, consecutive in g and `stride` doubles apart in
// shared memory.
TAG_DEV void copy_in_blocks(double* smem, int stride, const double* __restrict__ g, int count,
                            int ne) {
  const u32 s = (u32)__cvta_generic_to_shared(smem);
  if (((((size_t)g) | s | (count * 8u) | (stride * 8u)) & 15u) == 0) {
    const int c2 = count / 2;
    for (int t = threadIdx.x; t < ne * c2; t += blockDim.x) {
      const int el = t / c2, r = t - el * c2;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s + 8 * stride * el + 16 * r),
                   "l"(g + 2 * t));
    }
  } else {
    for (int t = threadIdx.x; t < ne * count; t += blockDim.x) {
      const int el = t / count, r = t - el * count;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s + 8 * (stride * el + r)),
                   "l"(g + t));
    }
  }
}
TAG_DEV void copy_in_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
TAG_DEV void copy_out(double* __restrict__ g, const double* smem, int count) {
  if (((((size_t)g) | (size_t)smem | (count * 8u)) & 15u) == 0) {
    for (int t = threadIdx.x; t < count / 2; t += blockDim.x)
      reinterpret_cast<double2*>(g)[t] = reinterpret_cast<const double2*>(smem)[t];
  } else {
    for (int t = threadIdx.x; t < count; t += blockDim.x) g[t] = smem[t];
  }
}

// Atomic max of a non-negative double stored as its IEEE bit pattern.
TAG_DEV void atomic_max_nonneg(double* addr, double v) {
  atomicMax(reinterpret_cast<unsigned long long*>(addr),
            static_cast<unsigned long long>(__double_as_longlong(v)));
}

// Carpenter-Kennedy RK4(3)5[2N] coefficients (NASA TM-109112, 1994).
struct CK2N54 {
  double A[5], B[5], c[5];
};

__host__ __device__ inline CK2N54 ck2n54() {
  return CK2N54{{0.0, -567301805773.0 / 1357537059087.0, -2404267990393.0 / 2016746695238.0,
                 -3550918686646.0 / 2091501179385.0, -1275806237668.0 / 842570457699.0},
                {1432997174477.0 / 9575080441755.0, 5161836677717.0 / 13612068292357.0,
                 1720146321549.0 / 2090206949498.0, 3134564353537.0 / 4481467310338.0,
                 2277821191437.0 / 14882151754819.0},
                {0.0, 1432997174477.0 / 9575080441755.0, 2526269341429.0 / 6820363962896.0,
                 2006345519317.0 / 3224310063776.0, 2802321613138.0 / 2924317926251.0}};
}

// One stage of a time integrator in the form the element kernels apply:
//   2N (ssp = 0):  k = A k + dt du,  u = u + B k
//   SSP (ssp = 1): w = u + (B dt) du,  u = A k + C w  (u = w where A = 0),
//                  k = u at the first stage (save), the step's starting state.
// The SSP schemes are the Shu-Osher forms of SSPRK43 (Kraaijevanger 1991;
// h = dt/2: u1 = u + h L(u), u2 = u1 + h L(u1), u3 = 2/3 u + 1/3 (u2 + h L(u2)),
// u_new = u3 + h L(u3)) and SSPRK33 (Shu & Osher 1988: u1 = u + dt L(u),
// u2 = 3/4 u + 1/4 (u1 + dt L(u1)), u_new = 1/3 u + 2/3 (u2 + dt L(u2))).
struct StageCoef {
  double A, B, C, c;  // c: stage time fraction
  int ssp, save;
};

inline int rk_stages(int scheme) {
  return scheme == TAG_RK_SSPRK43 ? 4 : scheme == TAG_RK_SSPRK33 ? 3 : 5;
}

inline StageCoef rk_stage(int scheme, int s) {
  if (scheme == TAG_RK_SSPRK43) {
    static const double c[4] = {0.0, 0.5, 1.0, 0.5};
    if (s == 2) return StageCoef{2.0 / 3.0, 0.5, 1.0 / 3.0, c[s], 1, 0};
    return StageCoef{0.0, 0.5, 1.0, c[s], 1, s == 0};
  }
  if (scheme == TAG_RK_SSPRK33) {
    static const double c[3] = {0.0, 1.0, 0.5};
    if (s == 1) return StageCoef{0.75, 1.0, 0.25, c[s], 1, 0};
    if (s == 2) return StageCoef{1.0 / 3.0, 1.0, 2.0 / 3.0, c[s], 1, 0};
    return StageCoef{0.0, 1.0, 1.0, c[s], 1, 1};
  }
  const CK2N54 ck = ck2n54();
  return StageCoef{ck.A[s], ck.B[s], 0.0, ck.c[s], 0, 0};
}

// Step control shared by all ensemble members (device memory, so a captured
// graph picks up new values without re-instantiation).
struct StepCtl {
  double cfl;
  double fixed_dt;
};

// Per-member step scalars, each an array of nmembers doubles in device memory.
struct MemberScalars {
  double* t;          // start time of the current step
  double* dt;         // current step size
  double* max_speed;  // running max over elements of (max lambda1 + max lambda2)
};

}  // namespace tag
