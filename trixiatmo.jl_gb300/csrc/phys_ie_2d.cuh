// Device physics of CompressibleEulerInternalEnergyEquationsWithGravity2D
// (reference: src/equations/compressible_euler_internal_energy_with_gravity_2d.jl).
// State u = (rho, rho_v1, rho_v2, rho_e_internal, phi), p = (gamma - 1) rho_e_internal;
// phi = g z is passive, so kernels evolve NA = 4 variables.  Volume flux
// (flux_conservative_etec :110-136, flux_nonconservative_etec :144-165);
// surface flux (flux_conservative_es :174-216, flux_nonconservative_es
// :224-246), whose nonconservative part differs on the two sides of an
// interface (kSurfaceNoncons); slip walls :77-99.
#pragma once
#include "tag_common.cuh"

namespace tag {

struct PhysIE2D {
  static constexpr int NV = 5;
  static constexpr int NA = 4;
  // rho/2, v1/2, v2/2, p/2, phi/2, theta = (p/rho) / (2 (gamma - 1)),
  // log2(rho), log2(p/rho) (log2_fixed words), pad (odd stride)
  static constexpr int NQ = 9;
  static constexpr bool kLastHalved = false;
  static constexpr bool kFixed = false;  // volume integral in FP64
  static constexpr bool kHasSources = false;
  static constexpr bool kSurfaceNoncons = true;

  struct Params {
    double gamma, gm1, inv_gm1;
  };

  // params = (c_p, c_v, g)
  static Params make_params(const double* p) {
    Params q;
    q.gamma = p[0] / p[1];
    q.gm1 = q.gamma - 1.0;
    q.inv_gm1 = 1.0 / (q.gamma - 1.0);
    return q;
  }

  TAG_DEV static void node_prims(const Params& P, const double* u, double* q, unsigned& bad) {
    const double rho = u[0];
    const double irho = int_rcp(rho), hir = 0.5 * irho;
    const double p = P.gm1 * u[3];
    const double pr = p * irho;
    q[0] = 0.5 * rho;
    q[1] = u[1] * hir;
    q[2] = u[2] * hir;
    q[3] = 0.5 * p;
    q[4] = 0.5 * u[4];
    q[5] = invertible(0.5 * pr * P.inv_gm1);
    q[6] = log_word(rho);
    q[7] = log_word(pr);
    if (not_positive(rho)) bad |= TAG_S_NEG_DENSITY;
    if (not_positive(p)) bad |= TAG_S_NEG_PRESSURE;
  }

  // flux_conservative_etec + half of flux_nonconservative_etec (antisymmetric)
  // on the halved node quantities; p_ll p_rr inv_ln_mean(rho_ll p_rr, rho_rr p_ll)
  // is evaluated as the equal inv_ln_mean(rho_ll/p_ll, rho_rr/p_rr), the mean
  // of the reciprocals of p/rho.
  TAG_DEV static void volume_pair(const Params& P, const double* qa, const double* qb, double n1,
                                  double n2, double* Fa, double* Fb) {
    const double rho_mean = (qa[0] + qb[0]) * ln_factor(qa[0], qb[0], log_difference(qa[6], qb[6]));
    const double e_mean = (qa[5] + qb[5]) * inv_ln_factor(qa[5], qb[5], log_difference(qa[7], qb[7]));
    const double v1 = qa[1] + qb[1], v2 = qa[2] + qb[2];  // averages
    const double vn = n1 * v1 + n2 * v2;                    // 0.5 (vn_a + vn_b)
    const double p_avg = qa[3] + qb[3];
    const double f1 = rho_mean * vn;
    const double g = qb[4] - qa[4];                  // (phi_b - phi_a) / 2
    const double pp = fma(rho_mean, g, p_avg), pm = fma(-rho_mean, g, p_avg);
    const double t1 = f1 * v1, t2 = f1 * v2;
    const double f4 = fma(f1, e_mean, p_avg * vn);
    const double dp = qb[3] - qa[3];                 // gp = -vn_avg (p_b - p_a) / 2
    Fa[0] = Fb[0] = f1;
    Fa[1] = fma(n1, pp, t1);
    Fb[1] = fma(n1, pm, t1);
    Fa[2] = fma(n2, pp, t2);
    Fb[2] = fma(n2, pm, t2);
    Fa[3] = fma(-vn, dp, f4);
    Fb[3] = fma(vn, dp, f4);
  }

  // interface speed of sound and normal velocity of the es pair
  TAG_DEV static double v_interface(const Params& P, const double* ul, const double* ur,
                                    double n1, double n2, double& vnl, double& vnr, double& pl,
                                    double& pr, double& a, double& nrm) {
    const double rl = ul[0], rr = ur[0];
    pl = P.gm1 * ul[3];
    pr = P.gm1 * ur[3];
    const double irl = int_rcp(rl), irr = int_rcp(rr);
    vnl = fma(ul[2], n2, ul[1] * n1) * irl;
    vnr = fma(ur[2], n2, ur[1] * n1) * irr;
    const double cl = int_sqrt(P.gamma * pl * irl), cr = int_sqrt(P.gamma * pr * irr);
    a = 0.5 * (cl + cr);
    nrm = int_sqrt(n1 * n1 + n2 * n2);
    return 0.5 * (vnl + vnr) - int_rcp(a * (rl + rr)) * (pr - pl) * nrm;
  }

  // flux_conservative_es
  TAG_DEV static void surface_flux(const Params& P, const double* ul, const double* ur, double n1,
                                   double n2, double* F) {
    double vnl, vnr, pl, pr, a, nrm;
    const double v_int = v_interface(P, ul, ur, n1, n2, vnl, vnr, pl, pr, a, nrm);
    const double rl = ul[0], rr = ur[0];
    const double rho_mean = ln_mean_of(rl, rr);
    const double rho_avg = 0.5 * (rl + rr);
    const double p_int = 0.5 * (pl + pr) - 0.5 * a * rho_avg * (vnr - vnl) * int_rcp(nrm);
    const double p_avg = 0.5 * (pl + pr);
    double rho_up, f2, f3;
    if (v_int >= 0.0) {
      rho_up = rho_mean - 0.5 * (rr - rl);
      f2 = ul[1] * v_int;
      f3 = ul[2] * v_int;
    } else {
      rho_up = rho_mean + 0.5 * (rr - rl);
      f2 = ur[1] * v_int;
      f3 = ur[2] * v_int;
    }
    const double inv_rho_p_mean =
        inv_ln_mean_of_reciprocals(pl * int_rcp(rl), pr * int_rcp(rr));
    const double f1 = rho_up * v_int;
    F[0] = f1;
    F[1] = f2 + p_int * n1;
    F[2] = f3 + p_int * n2;
    F[3] = f1 * inv_rho_p_mean * P.inv_gm1 + p_avg * v_int;
  }

  // flux_nonconservative_es of (ul, ur) along the primary's normal
  TAG_DEV static void surface_noncons(const Params& P, const double* ul, const double* ur,
                                      double n1, double n2, double* G) {
    double vnl, vnr, pl, pr, a, nrm;
    const double v_int = v_interface(P, ul, ur, n1, n2, vnl, vnr, pl, pr, a, nrm);
    G[0] = G[1] = G[2] = 0.0;
    G[3] = -v_int * (pr - pl);
  }

  // boundary_condition_slip_wall (outward normal): flux + 1/2 nonconservative
  // flux of the inner and the mirrored state
  TAG_DEV static void boundary_flux(const Params& P, const double* ui, double n1, double n2, int,
                                    int, double* F) {
    const double inn = int_rsqrt(n1 * n1 + n2 * n2);
    const double nx = n1 * inn, ny = n2 * inn;
    const double un = nx * ui[1] + ny * ui[2];
    const double ub[5] = {ui[0], ui[1] - 2.0 * un * nx, ui[2] - 2.0 * un * ny, ui[3], ui[4]};
    double G[4];
    surface_flux(P, ui, ub, n1, n2, F);
    surface_noncons(P, ui, ub, n1, n2, G);
#pragma unroll
    for (int v = 0; v < 4; ++v) F[v] += 0.5 * G[v];
  }

  TAG_DEV static void max_speeds(const Params& P, const double* u, double& l1, double& l2) {
    const double irho = int_rcp(u[0]);
    const double v1 = u[1] * irho, v2 = u[2] * irho;
    const double c = int_sqrt(P.gamma * (P.gm1 * u[3]) * irho);
    l1 = fabs(v1) + c;
    l2 = fabs(v2) + c;
  }
};

}  // namespace tag
