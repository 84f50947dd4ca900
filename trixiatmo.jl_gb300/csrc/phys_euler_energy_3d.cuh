// Device physics of CompressibleEulerEnergyEquationsWithGravity3D
// (reference: src/equations/compressible_euler_energy_with_gravity_3d.jl) and
// the Coriolis source (src/equations/initial_condition_compressible_euler_3d.jl:245-269).
// State u = (rho, rho_v1, rho_v2, rho_v3, rho_e, phi); phi is passive, so
// kernels evolve NA = 5 active variables.
#pragma once
#include "fixed_flux.cuh"

namespace tag {

struct PhysEnergy3D {
  static constexpr int NV = 6;
  static constexpr int NA = 5;
  // rho/2, v1/2, v2/2, v3/2, p/2, phi/4 (less the first node's), theta = (p/rho) / (4 (gamma - 1)),
  // log2(rho), log2(p/rho) (log2_fixed words; odd stride)
  static constexpr int NQ = 9;
  // volume_pair returns half the energy flux (the kernel doubles the node sums)
  static constexpr bool kLastHalved = true;
  static constexpr bool kFixed = true;  // volume integral in words (fixed_flux.cuh)
  static constexpr bool kHasSources = true;  // Coriolis, added per (node, variable)

  struct Params {
    double gamma, gm1, inv_gm1, c_lmars, quarter_c, inv_c, omega, quarter_inv_gm1;
  };

  static Params make_params(const double* p) {
    Params q;
    q.gamma = p[0] / p[1];
    q.gm1 = q.gamma - 1.0;
    q.inv_gm1 = 1.0 / (q.gamma - 1.0);
    q.quarter_inv_gm1 = 0.25 * q.inv_gm1;
    q.c_lmars = p[3];
    q.quarter_c = 0.25 * p[3];
    q.inv_c = 1.0 / p[3];
    q.omega = p[4];
    return q;
  }

  // cons2prim (:568-578) once per node, the reciprocal and both logarithms on
  // the integer pipe.
  TAG_HD static void node_prims(const Params& P, const double* u, double* q, unsigned& bad) {
    const double rho = u[0];
    const double ir = int_rcp(rho), hir = 0.5 * ir;
    const double m2 = fma(u[3], u[3], fma(u[2], u[2], u[1] * u[1]));
    const double p = P.gm1 * fma(-hir, m2, u[4]);
    const double pr = p * ir;
    q[0] = 0.5 * rho;
    q[1] = u[1] * hir;
    q[2] = u[2] * hir;
    q[3] = u[3] * hir;
    q[4] = 0.5 * p;
    q[5] = 0.25 * u[5];
    q[6] = invertible(pr * P.quarter_inv_gm1);
    q[7] = log_word(rho);
    q[8] = log_word(pr);
    if (not_positive(rho)) bad |= TAG_S_NEG_DENSITY;
    if (not_positive(p)) bad |= TAG_S_NEG_PRESSURE;
  }

  // flux_ranocha (3D, :382-415) + half of flux_nonconservative_waruszewski_etal
  // (3D, :135-159) for one symmetric pair; see PhysEnergy2D::volume_pair.
  // nrm is twice the average of the two nodes' contravariant vectors (D_split
  // is halved).  p_ll p_rr inv_ln_mean(rho_ll p_rr, rho_rr p_ll) is
  // inv_ln_mean(rho_ll/p_ll, rho_rr/p_rr), the mean of the reciprocals of the
  // node values p/rho.  With g = (phi_b - phi_a) / 4 the momentum fluxes of the
  // two sides are f1 v + n (p_avg +- 2 rho_mean g), and half the energy fluxes
  //   f1 (v_a.v_b / 4 + mean(p/rho) / (2 (gamma - 1)) +- g) + (p_a vn_b + p_b vn_a) / 4.
  // The FP64 pipe bounds the kernel, so the reciprocal and the two series of
  // the means go to the integer pipe (int_math.cuh): the right-hand side of
  // the 2,654,208-node shell at polydeg 5 went from 3.48 to 2.32 ms.  Elements
  // in range take fx_energy_pair (fixed_flux.cuh) instead of this form.
  TAG_HD static void volume_pair(const Params& P, const double* qa, const double* qb,
                                 const double* nrm, double* Fa, double* Fb) {
    const double R = ln_factor(qa[0], qb[0], log_difference(qa[7], qb[7]));
    const double Q = inv_ln_factor(qa[6], qb[6], log_difference(qa[8], qb[8]));
    const double rho_mean = (qa[0] + qb[0]) * R;
    const double n1 = nrm[0], n2 = nrm[1], n3 = nrm[2];
    const double v1 = qa[1] + qb[1], v2 = qa[2] + qb[2], v3 = qa[3] + qb[3];
    // halved normal velocities of both nodes: vn = 0.5 (vn_a + vn_b)
    const double vna = fma(qa[3], n3, fma(qa[2], n2, qa[1] * n1));
    const double vnb = fma(qb[3], n3, fma(qb[2], n2, qb[1] * n1));
    const double f1 = rho_mean * (vna + vnb);
    const double g = qb[5] - qa[5];
    const double p_avg = qa[4] + qb[4], r2 = twice(rho_mean);
    const double pp = fma(r2, g, p_avg), pm = fma(-r2, g, p_avg);
    const double t1 = f1 * v1, t2 = f1 * v2, t3 = f1 * v3;
    Fa[0] = f1;
    Fb[0] = f1;
    Fa[1] = fma(n1, pp, t1);
    Fb[1] = fma(n1, pm, t1);
    Fa[2] = fma(n2, pp, t2);
    Fb[2] = fma(n2, pm, t2);
    Fa[3] = fma(n3, pp, t3);
    Fb[3] = fma(n3, pm, t3);
    const double vv = fma(qa[3], qb[3], fma(qa[2], qb[2], qa[1] * qb[1]));
    const double x = fma(qa[6] + qb[6], Q, vv);
    const double e = fma(f1, x, fma(qa[4], vnb, qb[4] * vna));
    Fa[4] = fma(f1, g, e);
    Fb[4] = fma(-f1, g, e);
  }

  TAG_HD static void fixed_pair(const Params&, const double* qa, const double* qb,
                                const double* na, const double* nb, u64 Q, const FxShift& k,
                                i64* Fa, i64* Fb) {
    fx_energy_pair<3>(reinterpret_cast<const i64*>(qa), reinterpret_cast<const i64*>(qb),
                      reinterpret_cast<const i64*>(na), reinterpret_cast<const i64*>(nb), Q, k, Fa,
                      Fb);
  }

  // FluxLMARS (3D, :430-466) for the (unnormalised) normal n:
  //   p = (p_ll + p_rr)/2 - c rho (v_rr - v_ll) / (2 |n|),
  //   v = (v_ll + v_rr)/2 - (p_rr - p_ll) |n| / (2 c rho),  rho = (rho_ll + rho_rr)/2,
  // the reciprocals and the reciprocal root on the integer pipe, and
  // p = (gamma - 1)(rho e - |rho v|^2 / (2 rho)).
  TAG_DEV static void lmars(const Params& P, const double* ul, const double* ur, const double* n,
                            double* F) {
    const double rho_ll = ul[0], rho_rr = ur[0];
    const double srho = rho_ll + rho_rr;
    const double irl = int_rcp(rho_ll), irr = int_rcp(rho_rr), isum = int_rcp(srho);
    const double ml = fma(ul[3], ul[3], fma(ul[2], ul[2], ul[1] * ul[1]));
    const double mr = fma(ur[3], ur[3], fma(ur[2], ur[2], ur[1] * ur[1]));
    const double pl = P.gm1 * fma(-0.5 * irl, ml, ul[4]);
    const double pr = P.gm1 * fma(-0.5 * irr, mr, ur[4]);
    const double vl = fma(ul[3], n[2], fma(ul[2], n[1], ul[1] * n[0])) * irl;
    const double vr = fma(ur[3], n[2], fma(ur[2], n[1], ur[1] * n[0])) * irr;
    const double nsq = fma(n[2], n[2], fma(n[1], n[1], n[0] * n[0]));
    const double inorm = int_rsqrt(nsq), norm_ = nsq * inorm;
    const double p = 0.5 * (pl + pr) - P.quarter_c * srho * (vr - vl) * inorm;
    const double v = 0.5 * (vl + vr) - P.inv_c * (pr - pl) * norm_ * isum;
    const double* us = v >= 0.0 ? ul : ur;
    const double ps = v >= 0.0 ? pl : pr;
    F[0] = v * us[0];
    F[1] = v * us[1] + p * n[0];
    F[2] = v * us[2] + p * n[1];
    F[3] = v * us[3] + p * n[2];
    F[4] = v * us[4] + ps * v;
  }

  TAG_DEV static void surface_flux(const Params& P, const double* ul, const double* ur,
                                   const double* n, double* F) {
    lmars(P, ul, ur, n, F);
  }

  // boundary_condition_slip_wall (3D), :93-116, with the outward normal n: the
  // LMARS flux against the mirrored state, whose normal velocity is the opposite
  // and whose density and pressure are the same, so only the pressure
  // p + c rho v_n / |n| stays.  (Formed through the mirrored state, its rounding
  // is a flux through the wall, which the end weights raise to the largest error
  // of the density: 0.7 before and 0.4 now of the FP64 kernels' on shells of four
  // layers.)
  TAG_DEV static void boundary_flux(const Params& P, const double* ui, const double* n, double* F) {
    const double m2 = fma(ui[3], ui[3], fma(ui[2], ui[2], ui[1] * ui[1]));
    const double p = P.gm1 * fma(-0.5 * int_rcp(ui[0]), m2, ui[4]);
    const double mn = fma(ui[3], n[2], fma(ui[2], n[1], ui[1] * n[0]));
    const double inorm = int_rsqrt(fma(n[2], n[2], fma(n[1], n[1], n[0] * n[0])));
    const double pw = fma(P.c_lmars * inorm, mn, p);
    F[0] = F[4] = 0.0;
    F[1] = pw * n[0];
    F[2] = pw * n[1];
    F[3] = pw * n[2];
  }

  // coriolis_source: du2 += 2 Omega rho_v2, du3 -= 2 Omega rho_v1
  TAG_DEV static double source(const Params& P, const double* u, int v) {
    if (v == 1) return 2.0 * P.omega * u[2];
    if (v == 2) return -2.0 * P.omega * u[1];
    return 0.0;
  }

  TAG_DEV static void max_speeds(const Params& P, const double* u, double* l) {
    const double irho = int_rcp(u[0]);
    const double v1 = u[1] * irho, v2 = u[2] * irho, v3 = u[3] * irho;
    const double p = P.gm1 * (u[4] - 0.5 * (u[1] * v1 + u[2] * v2 + u[3] * v3));
    const double c = int_sqrt(P.gamma * p * irho);
    l[0] = fabs(v1) + c;
    l[1] = fabs(v2) + c;
    l[2] = fabs(v3) + c;
  }
};

}  // namespace tag
