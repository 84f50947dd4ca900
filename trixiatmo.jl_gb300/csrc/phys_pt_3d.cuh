// Device physics of CompressibleEulerPotentialTemperatureEquationsWithGravity3D
// (reference: src/equations/compressible_euler_potential_temperature_gravity_3d.jl)
// with the Coriolis source (src/equations/initial_condition_compressible_euler_3d.jl:245-269).
// State u = (rho, rho_v1, rho_v2, rho_v3, rho_theta, phi), p = K rho_theta^gamma;
// phi = g z is passive, so kernels evolve NA = 5 variables.  Volume fluxes
// flux_tec / flux_ec / flux_etec (:428-533) with the nonconservative gravity
// term of Waruszewski et al. (or Artiano et al., Souza et al.; :146-211);
// surface flux (FluxLMARS(c), flux_zero) (:213-256); slip walls (:83-107).
// The means as in phys_pt_2d.cuh.
#pragma once
#include "phys_pt_2d.cuh"

namespace tag {

struct PhysPT3D {
  static constexpr int NV = 6;
  static constexpr int NA = 5;
  // rho/2, v1/2, v2/2, v3/2, p/2, phi/2, rho_theta/2, the third mean's half
  // value (phys_pt_2d.cuh), log2(rho), log2(rho_theta), (pad: odd stride)
  static constexpr int NQ = 11;
  static constexpr bool kLastHalved = false;
  static constexpr bool kFixed = false;  // volume integral in FP64
  static constexpr bool kHasSources = true;  // Coriolis, per (node, variable)

  struct Params {
    PhysPT2D::Params pt;  // gamma, K, LMARS c, Stolarsky series, volume / gravity-term kinds
    double omega;
  };

  // params = (c_p, c_v, g, LMARS c, nonconservative kind, volume kind, Omega)
  static Params make_params(const double* p) {
    double p2[8];
    for (int k = 0; k < 8; ++k) p2[k] = p[k];
    p2[6] = 0.0;  // surface (FluxLMARS(c), flux_zero)
    p2[7] = 0.0;
    Params q;
    q.pt = PhysPT2D::make_params(p2);
    q.omega = p[6];
    return q;
  }

  TAG_DEV static void node_prims(const Params& Q, const double* u, double* q, unsigned& bad) {
    const PhysPT2D::Params& P = Q.pt;
    const double rho = u[0];
    const double irho = int_rcp(rho), hir = 0.5 * irho;
    q[0] = 0.5 * rho;
    q[1] = u[1] * hir;
    q[2] = u[2] * hir;
    q[3] = u[3] * hir;
    q[4] = 0.5 * PhysPT2D::pressure(P, u[4]);
    q[5] = 0.5 * u[5];
    q[6] = invertible(0.5 * u[4]);
    q[7] = PhysPT2D::third_value(P, rho, u[4], irho);
    q[8] = log_word(rho);
    q[9] = log_word(u[4]);
    if (not_positive(rho)) bad |= TAG_S_NEG_DENSITY;
    if (not_positive(u[4])) bad |= TAG_S_NEG_PRESSURE;
  }

  // One symmetric pair: the two-point flux F plus half the nonconservative
  // term G (antisymmetric in the pair): Fa = F + G/2, Fb = F - G/2.
  // (flux_kennedy_gruber, :333-359: arithmetic means of rho, v, p and theta)
  TAG_DEV static void volume_pair(const Params& Q, const double* a, const double* b,
                                  const double* nrm, double* Fa, double* Fb) {
    const PhysPT2D::Params& P = Q.pt;
    const double n1 = nrm[0], n2 = nrm[1], n3 = nrm[2];
    const double v1 = a[1] + b[1], v2 = a[2] + b[2], v3 = a[3] + b[3];
    const double vn = n1 * v1 + n2 * v2 + n3 * v3;
    double f1, f5, ravg;
    PhysPT2D::mean_fluxes(P, a[0], b[0], a[6], b[6], a[7], b[7], log_difference(a[8], b[8]),
                          log_difference(a[9], b[9]), vn, f1, f5, ravg);
    const double pa = a[4] + b[4];
    const double g = b[5] - a[5];  // (phi_b - phi_a) / 2
    const double pp = fma(ravg, g, pa), pm = fma(-ravg, g, pa);
    const double t1 = f1 * v1, t2 = f1 * v2, t3 = f1 * v3;
    Fa[0] = Fb[0] = f1;
    Fa[1] = fma(n1, pp, t1);
    Fb[1] = fma(n1, pm, t1);
    Fa[2] = fma(n2, pp, t2);
    Fb[2] = fma(n2, pm, t2);
    Fa[3] = fma(n3, pp, t3);
    Fb[3] = fma(n3, pm, t3);
    Fa[4] = Fb[4] = f5;
  }

  // FluxLMARS (:213-256)
  TAG_DEV static void lmars(const Params& Q, const double* ul, const double* ur, const double* n,
                            double* F) {
    const PhysPT2D::Params& P = Q.pt;
    const double a = P.c_lmars;
    const double p_l = PhysPT2D::pressure(P, ul[4]), p_r = PhysPT2D::pressure(P, ur[4]);
    const double v_l = fma(ul[3], n[2], fma(ul[2], n[1], ul[1] * n[0])) * int_rcp(ul[0]);
    const double v_r = fma(ur[3], n[2], fma(ur[2], n[1], ur[1] * n[0])) * int_rcp(ur[0]);
    const double nsq = fma(n[2], n[2], fma(n[1], n[1], n[0] * n[0]));
    const double inorm = int_rsqrt(nsq), nrm = nsq * inorm;
    const double rs = ul[0] + ur[0];  // 2 rho
    const double p_int = 0.5 * (p_l + p_r) - 0.25 * a * rs * (v_r - v_l) * inorm;
    const double v_int = 0.5 * (v_l + v_r) - int_rcp(a * rs) * (p_r - p_l) * nrm;
    const double* us = v_int > 0.0 ? ul : ur;
    F[0] = us[0] * v_int;
    F[1] = us[1] * v_int + p_int * n[0];
    F[2] = us[2] * v_int + p_int * n[1];
    F[3] = us[3] * v_int + p_int * n[2];
    F[4] = us[4] * v_int;
  }

  TAG_DEV static void surface_flux(const Params& Q, const double* ul, const double* ur,
                                   const double* n, double* F) {
    lmars(Q, ul, ur, n, F);
  }

  // boundary_condition_slip_wall (:83-107) with the outward normal n: the LMARS
  // flux against the mirrored state, of which only the pressure p + c rho v_n / |n|
  // stays (see PhysEnergy3D::boundary_flux)
  TAG_DEV static void boundary_flux(const Params& Q, const double* ui, const double* n, double* F) {
    const PhysPT2D::Params& P = Q.pt;
    const double mn = fma(ui[3], n[2], fma(ui[2], n[1], ui[1] * n[0]));
    const double inorm = int_rsqrt(fma(n[2], n[2], fma(n[1], n[1], n[0] * n[0])));
    const double pw = fma(P.c_lmars * inorm, mn, PhysPT2D::pressure(P, ui[4]));
    F[0] = F[4] = 0.0;
    F[1] = pw * n[0];
    F[2] = pw * n[1];
    F[3] = pw * n[2];
  }

  // coriolis_source: du2 += 2 Omega rho_v2, du3 -= 2 Omega rho_v1
  TAG_DEV static double source(const Params& Q, const double* u, int v) {
    if (v == 1) return 2.0 * Q.omega * u[2];
    if (v == 2) return -2.0 * Q.omega * u[1];
    return 0.0;
  }

  // max_abs_speeds (:695-700)
  TAG_DEV static void max_speeds(const Params& Q, const double* u, double* l) {
    const PhysPT2D::Params& P = Q.pt;
    const double irho = int_rcp(u[0]);
    const double v1 = u[1] * irho, v2 = u[2] * irho, v3 = u[3] * irho;
    const double c = int_sqrt(P.gamma * PhysPT2D::pressure(P, u[4]) * irho);
    l[0] = fabs(v1) + c;
    l[1] = fabs(v2) + c;
    l[2] = fabs(v3) + c;
  }
};

}  // namespace tag
