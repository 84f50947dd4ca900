// Device physics of CompressibleEulerPotentialTemperatureEquationsWithGravity2D
// (reference: src/equations/compressible_euler_potential_temperature_gravity_2d.jl).
// State u = (rho, rho_v1, rho_v2, rho_theta, phi), p = K rho_theta^gamma; phi = g z
// is passive, so kernels evolve NA = 4 variables.  Volume fluxes flux_tec /
// flux_ec / flux_etec with the nonconservative gravity term of Waruszewski et al.
// (or Artiano et al., Souza et al.); surface flux (FluxLMARS(c), flux_zero).
//
// The Stolarsky mean S(x, y) = (gamma-1)/gamma (y^g - x^g) / (y^(g-1) - x^(g-1))
// (Winters et al. 2020) is (x+y)/2 times an even function of log(y/x), evaluated
// as its series on the integer pipe for values within a factor of two and from
// exponentials of the logarithms' difference up to 256 (int_math.cuh); beyond
// that, and for gamma outside (1, 2), from powers.
#pragma once
#include "tag_common.cuh"

namespace tag {

struct PhysPT2D {
  static constexpr int NV = 5;
  static constexpr int NA = 4;
  // rho/2, v1/2, v2/2, p/2, phi/2, rho_theta/2, the third mean's half value
  // (flux_ec: theta = rho_theta/rho, flux_etec: 1/theta), log2(rho),
  // log2(rho_theta) (log2_fixed words; odd stride)
  static constexpr int NQ = 9;
  static constexpr bool kLastHalved = false;
  static constexpr bool kFixed = false;  // volume integral in FP64
  // MountainWaveSetup's Rayleigh damping when set (Params::mountain)
  static constexpr bool kHasSources = true;
  // surface flux (FluxLMARS(c), flux_zero) or (flux_ec, a nonconservative
  // gravity term); the interface kernel adds the per-side term when snc >= 0
  static constexpr bool kSurfaceNoncons = true;

  struct Params {
    double gamma, K, c_lmars, stol_fac;  // stol_fac = (gamma - 1) / gamma
    double sc[8];                        // Stolarsky series in f^2 (gamma outside (1, 2))
    EvenSeries stol;                     // Stolarsky factor of the logarithms' difference
    u64 gamma_q61;                       // gamma as int_pow takes it
    u64 stol_q64;                        // 2 (gamma - 1) / gamma, 0: no middle range
    int volume;                          // 0 flux_tec, 1 flux_ec, 2 flux_etec,
                                         // 3 flux_kennedy_gruber (3D only)
    int nc;                              // 0 waruszewski, 1 artiano, 2 souza
    int surface;                         // 0 FluxLMARS(c), 1 flux_ec
    int snc;                             // surface gravity term: -1 none (flux_zero), else as nc
    int mountain;                        // 1: MountainWaveSetup's damping source
    double g;                            // gravity
    double mw[8];  // theta_0, u0, N, z_damping_start, z_damping_end, x_damping_start,
                   // x_damping_end, damping_rate
  };

  // params = (c_p, c_v, g, LMARS c, nonconservative kind, volume kind,
  // surface kind, surface nonconservative kind + 1)
  static Params make_params(const double* p) {
    Params q;
    const double c_p = p[0], c_v = p[1], R = c_p - c_v;
    q.gamma = c_p / c_v;
    q.K = 100000.0 * pow(R / 100000.0, q.gamma);
    q.c_lmars = p[3];
    q.stol_fac = (q.gamma - 1.0) / q.gamma;
    q.stol = stolarsky_series(q.gamma);
    q.gamma_q61 = pow_exponent(q.gamma);
    // (stolarsky_deficit_middle's range)
    q.stol_q64 = q.gamma >= 1.3 && q.gamma <= 1.9
                     ? (u64)ldexpl(2.0L * ((long double)q.gamma - 1.0L) / q.gamma, 64)
                     : 0;
    q.nc = (int)p[4];
    q.volume = (int)p[5];
    q.surface = (int)p[6];
    q.snc = (int)p[7] - 1;
    q.mountain = 0;
    q.g = p[2];
    for (int k = 0; k < 8; ++k) q.mw[k] = 0.0;
    double a[8], b[8];
    for (int j = 0; j < 8; ++j) {
      double ra = 1.0, rb = 1.0;
      for (int i = 0; i < 2 * j + 1; ++i) {
        ra = ra * (q.gamma - i) / (i + 1);
        rb = rb * (q.gamma - 1.0 - i) / (i + 1);
      }
      a[j] = ra / q.gamma;
      b[j] = rb / (q.gamma - 1.0);
    }
    for (int k = 0; k < 8; ++k) {
      double s = a[k];
      for (int i = 1; i <= k; ++i) s -= b[i] * q.sc[k - i];
      q.sc[k] = s;
    }
    return q;
  }

  TAG_DEV static double pressure(const Params& P, double rho_theta) {
    return P.K * int_pow(rho_theta, P.gamma, P.gamma_q61);
  }

  // the third mean's half node value (volume 3: flux_kennedy_gruber's theta)
  TAG_DEV static double third_value(const Params& P, double rho, double rho_theta, double irho) {
    if (P.volume == 0) return 0.0;
    if (P.volume == 2) return 0.5 * rho * int_rcp(rho_theta);
    const double x = 0.5 * rho_theta * irho;
    return P.volume == 1 ? invertible(x) : x;
  }

  TAG_DEV static void node_prims(const Params& P, const double* u, double* q, unsigned& bad) {
    const double rho = u[0];
    const double irho = int_rcp(rho), hir = 0.5 * irho;
    q[0] = 0.5 * rho;
    q[1] = u[1] * hir;
    q[2] = u[2] * hir;
    q[3] = 0.5 * pressure(P, u[3]);
    q[4] = 0.5 * u[4];
    q[5] = invertible(0.5 * u[3]);
    q[6] = third_value(P, rho, u[3], irho);
    q[7] = log_word(rho);
    q[8] = log_word(u[3]);
    if (not_positive(rho)) bad |= TAG_S_NEG_DENSITY;
    if (not_positive(u[3])) bad |= TAG_S_NEG_PRESSURE;
  }

  // Stolarsky mean over the arithmetic mean beyond a factor of two: up to 256
  // from the logarithms' difference (a: its magnitude), else from the values
  // themselves, the series in f^2 where they nearly agree (gamma outside (1, 2)),
  // else powers
  static __device__ __noinline__ double stolarsky_factor_far(const Params& P, double x, double y,
                                                             u64 a) {
    if (opposite_signs(x, y)) return quiet_nan();
    if (P.stol.ok && P.stol_q64 && middle_range(a))
      return middle_factor(stolarsky_deficit_middle(a, P.gamma_q61, P.stol_q64));
    const double s = x + y, d = y - x;
    const double t = d / s, f2 = t * t;
    if (f2 < 1e-2) {
      double r = P.sc[7];
      for (int k = 6; k >= 0; --k) r = fma(r, f2, P.sc[k]);
      return r;
    }
    const double xg = pow(x, P.gamma), yg = pow(y, P.gamma);
    return 2.0 * (P.stol_fac * (yg - xg) / (yg / y - xg / x)) / s;
  }
  // x, y: the values or their halves (the factor is homogeneous)
  TAG_DEV static double stolarsky_factor(const Params& P, double x, double y, i64 d) {
    const u64 a = magnitude(d);
    return series_in_range(a) && P.stol.ok ? even_factor(P.stol, log_square(a))
                                           : stolarsky_factor_far(P, x, y, a);
  }
  TAG_DEV static double stolarsky(const Params& P, double x, double y) {
    return 0.5 * (x + y) * stolarsky_factor(P, x, y, log2_fixed(y) - log2_fixed(x));
  }

  // The mass flux f1, the rho_theta flux f and the density average of the
  // gravity term for the averaged normal velocity vn, from the node values
  // rho/2, rho_theta/2, the third value and the logarithms' differences.
  TAG_DEV static void mean_fluxes(const Params& P, double ra, double rb, double ta, double tb,
                                  double xa, double xb, i64 dr, i64 dt, double vn, double& f1,
                                  double& f, double& ravg) {
    const double rs = ra + rb;
    double rho_ln = 0.0;
    if (P.volume == 1) {
      rho_ln = rs * ln_factor(ra, rb, dr);
      f1 = rho_ln * vn;
      f = f1 * ((xa + xb) * inv_ln_factor(xa, xb, dt - dr));
    } else if (P.volume == 3) {
      f1 = rs * vn;
      f = f1 * (xa + xb);
    } else {
      f = (ta + tb) * stolarsky_factor(P, ta, tb, dt) * vn;
      if (P.volume == 0) {
        rho_ln = rs * ln_factor(ra, rb, dr);
        f1 = rho_ln * vn;
      } else {
        f1 = f * ((xa + xb) * ln_factor(xa, xb, dr - dt));
      }
    }
    if (P.nc == 0) ravg = P.volume >= 2 ? rs * ln_factor(ra, rb, dr) : rho_ln;
    else if (P.nc == 1) ravg = rs * stolarsky_factor(P, ra, rb, dr);
    else ravg = rs;
  }

  // One symmetric pair: the two-point flux F plus half the nonconservative
  // term G (antisymmetric in the pair): Fa = F + G/2, Fb = F - G/2.
  TAG_DEV static void volume_pair(const Params& P, const double* a, const double* b, double n1,
                                  double n2, double* Fa, double* Fb) {
    const double v1 = a[1] + b[1], v2 = a[2] + b[2];
    const double vn = n1 * v1 + n2 * v2;
    double f1, f4, ravg;
    mean_fluxes(P, a[0], b[0], a[5], b[5], a[6], b[6], log_difference(a[7], b[7]),
                log_difference(a[8], b[8]), vn, f1, f4, ravg);
    const double pa = a[3] + b[3];
    const double g = b[4] - a[4];  // (phi_b - phi_a) / 2
    const double pp = fma(ravg, g, pa), pm = fma(-ravg, g, pa);
    const double t1 = f1 * v1, t2 = f1 * v2;
    Fa[0] = Fb[0] = f1;
    Fa[1] = fma(n1, pp, t1);
    Fb[1] = fma(n1, pm, t1);
    Fa[2] = fma(n2, pp, t2);
    Fb[2] = fma(n2, pm, t2);
    Fa[3] = Fb[3] = f4;
  }

  // FluxLMARS (:171-193)
  TAG_DEV static void lmars(const Params& P, const double* ul, const double* ur, double n1,
                            double n2, double* F) {
    const double a = P.c_lmars;
    const double p_l = pressure(P, ul[3]), p_r = pressure(P, ur[3]);
    const double v_l = fma(ul[2], n2, ul[1] * n1) * int_rcp(ul[0]);
    const double v_r = fma(ur[2], n2, ur[1] * n1) * int_rcp(ur[0]);
    const double nsq = fma(n2, n2, n1 * n1), inorm = int_rsqrt(nsq), nrm = nsq * inorm;
    const double rs = ul[0] + ur[0];  // 2 rho
    const double p_int = 0.5 * (p_l + p_r) - 0.25 * a * rs * (v_r - v_l) * inorm;
    const double v_int = 0.5 * (v_l + v_r) - int_rcp(a * rs) * (p_r - p_l) * nrm;
    const double* us = v_int > 0.0 ? ul : ur;
    F[0] = us[0] * v_int;
    F[1] = us[1] * v_int + p_int * n1;
    F[2] = us[2] * v_int + p_int * n2;
    F[3] = us[3] * v_int;
  }

  // flux_ec (:290-321) of full states
  TAG_DEV static void flux_ec(const Params& P, const double* ul, const double* ur, double n1,
                              double n2, double* F) {
    const double irl = int_rcp(ul[0]), irr = int_rcp(ur[0]);
    const double v1l = ul[1] * irl, v2l = ul[2] * irl, v1r = ur[1] * irr, v2r = ur[2] * irr;
    const double vn = 0.5 * ((v1l * n1 + v2l * n2) + (v1r * n1 + v2r * n2));
    const double pa = 0.5 * (pressure(P, ul[3]) + pressure(P, ur[3]));
    const double f1 = ln_mean_of(ul[0], ur[0]) * vn;
    const double inv_sig = inv_ln_mean_of_reciprocals(ul[3] * irl, ur[3] * irr);
    F[0] = f1;
    F[1] = f1 * 0.5 * (v1l + v1r) + pa * n1;
    F[2] = f1 * 0.5 * (v2l + v2r) + pa * n2;
    F[3] = f1 * inv_sig;
  }

  TAG_DEV static void surface_flux(const Params& P, const double* ul, const double* ur, double n1,
                                   double n2, double* F) {
    if (P.surface == 1)
      flux_ec(P, ul, ur, n1, n2, F);
    else
      lmars(P, ul, ur, n1, n2, F);
  }

  // the nonconservative gravity term of the surface flux, G(ul, ur) along the
  // primary's normal (zero for flux_zero)
  // MountainWaveSetup as source terms (src/equations/initial_condition_compressible_euler_2d.jl:174-200):
  // relaxation of v1 to u0, of v2 to 0 and of theta to theta_0 exp(N^2 z / g)
  // at the rate of rayleigh_damping_coefficient (:80-106), a sum of sin^2
  // ramps above z_damping_start and beyond +-x_damping_start
  TAG_DEV static void source(const Params& P, const double* u, const double* x, double,
                             double* s) {
    s[0] = s[1] = s[2] = s[3] = 0.0;
    if (!P.mountain) return;
    const double rate = P.mw[7], zs = P.mw[3], ze = P.mw[4], xs = P.mw[5], xe = P.mw[6];
    double dv = 0.0, dr = 0.0, dl = 0.0;
    if (x[1] > zs) {
      const double r = sinpi(int_div(0.5 * (x[1] - zs), ze - zs));
      dv = rate * (r * r);
    }
    if (!(x[0] < xs)) {
      const double r = sinpi(int_div(0.5 * (x[0] - xs), xe - xs));
      dr = rate * (r * r);
    }
    if (!(x[0] > -xs)) {
      const double r = sinpi(int_div(0.5 * (x[0] + xs), -xe + xs));
      dl = rate * (r * r);
    }
    const double damping = -(dv + dr + dl);
    const double irho = int_rcp(u[0]);
    const double v1 = u[1] * irho, theta = u[3] * irho;
    const double theta_b = P.mw[0] * int_exp(int_div(P.mw[2] * P.mw[2], P.g) * x[1]);
    s[1] = u[0] * (v1 - P.mw[1]) * damping;
    s[2] = u[2] * damping;
    s[3] = u[0] * (theta - theta_b) * damping;
  }

  TAG_DEV static void surface_noncons(const Params& P, const double* ul, const double* ur,
                                      double n1, double n2, double* G) {
    G[0] = G[1] = G[2] = G[3] = 0.0;
    if (P.snc < 0) return;
    double ra;
    if (P.snc == 0) {
      ra = ln_mean_of(ul[0], ur[0]);
    } else if (P.snc == 1) {
      ra = stolarsky(P, ul[0], ur[0]);
    } else {
      ra = 0.5 * (ul[0] + ur[0]);
    }
    const double jump = ur[4] - ul[4];
    G[1] = n1 * ra * jump;
    G[2] = n2 * ra * jump;
  }

  // Slip walls.  TAG_BC_SLIP_WALL_STRUCTURED (:62-83): reached with the normal
  // vector in the `orientation` slot, so rho_v2 is mirrored; states ordered by
  // the face parity; returned OUTWARD.  Otherwise (:45-60) the normal momentum
  // is mirrored about the outward normal (n1, n2).
  TAG_DEV static void boundary_flux(const Params& P, const double* ui, double n1, double n2,
                                    int face, int kind, double* F) {
    // (the wall's nonconservative term vanishes: both states carry the same phi)
    if (kind == TAG_BC_SLIP_WALL_STRUCTURED) {
      const double ub[5] = {ui[0], ui[1], -ui[2], ui[3], ui[4]};
      if (face & 1) {
        surface_flux(P, ui, ub, n1, n2, F);
      } else {
        surface_flux(P, ub, ui, n1, n2, F);
        F[0] = -F[0]; F[1] = -F[1]; F[2] = -F[2]; F[3] = -F[3];
      }
    } else {
      const double inn = int_rsqrt(n1 * n1 + n2 * n2);
      const double nx = n1 * inn, ny = n2 * inn;
      const double un = nx * ui[1] + ny * ui[2];
      const double ub[5] = {ui[0], ui[1] - 2.0 * un * nx, ui[2] - 2.0 * un * ny, ui[3], ui[4]};
      surface_flux(P, ui, ub, n1, n2, F);
    }
  }

  // max_abs_speeds
  TAG_DEV static void max_speeds(const Params& P, const double* u, double& l1, double& l2) {
    const double irho = int_rcp(u[0]);
    const double v1 = u[1] * irho, v2 = u[2] * irho;
    const double c = int_sqrt(P.gamma * pressure(P, u[3]) * irho);
    l1 = fabs(v1) + c;
    l2 = fabs(v2) + c;
  }
};

}  // namespace tag
