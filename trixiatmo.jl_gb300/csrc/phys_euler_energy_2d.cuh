// Device physics of CompressibleEulerEnergyEquationsWithGravity2D
// (reference: src/equations/compressible_euler_energy_with_gravity_2d.jl).
// State u = (rho, rho_v1, rho_v2, rho_e, phi); phi = g z is passive (zero flux,
// zero time derivative), so kernels evolve NA = 4 active variables.
#pragma once
#include "fixed_flux.cuh"

namespace tag {

struct PhysEnergy2D {
  static constexpr int NV = 5;  // stored variables per node
  static constexpr int NA = 4;  // variables with nonzero du
  // per-node quantities kept in shared memory (odd stride: no bank conflicts):
  // rho/2, v1/2, v2/2, p/2, phi/4 (less the first node's), theta = (p/rho) / (4 (gamma - 1)),
  // log2(rho), log2(p/rho) (log2_fixed words), (pad)
  static constexpr int NQ = 9;
  // volume_pair returns half the energy flux (the kernel doubles the node sums)
  static constexpr bool kLastHalved = true;
  static constexpr bool kFixed = true;  // volume integral in words (fixed_flux.cuh)
  static constexpr bool kHasSources = false;
  static constexpr bool kSurfaceNoncons = false;  // surface flux only (flux_zero)

  struct Params {
    double gamma, gm1, inv_gm1, c_lmars, quarter_c, inv_c, quarter_inv_gm1;
  };

  static Params make_params(const double* p) {
    Params q;
    const double c_p = p[0], c_v = p[1];
    q.gamma = c_p / c_v;
    q.gm1 = q.gamma - 1.0;
    q.inv_gm1 = 1.0 / (q.gamma - 1.0);
    q.c_lmars = p[3];
    q.quarter_c = 0.25 * p[3];
    q.inv_c = 1.0 / p[3];
    q.quarter_inv_gm1 = 0.25 * q.inv_gm1;
    return q;
  }

  // cons2prim (:527-536), once per node, the reciprocal and both logarithms
  // on the integer pipe; flags bad states.
  TAG_HD static void node_prims(const Params& P, const double* u, double* q, unsigned& bad) {
    const double rho = u[0];
    const double ir = int_rcp(rho), hir = 0.5 * ir;
    const double p = P.gm1 * fma(-hir, fma(u[2], u[2], u[1] * u[1]), u[3]);
    const double pr = p * ir;
    q[0] = 0.5 * rho;
    q[1] = u[1] * hir;
    q[2] = u[2] * hir;
    q[3] = 0.5 * p;
    q[4] = 0.25 * u[4];
    q[5] = invertible(pr * P.quarter_inv_gm1);
    q[6] = log_word(rho);
    q[7] = log_word(pr);
    if (not_positive(rho)) bad |= TAG_S_NEG_DENSITY;
    if (not_positive(p)) bad |= TAG_S_NEG_PRESSURE;
  }

  // One symmetric pair of the volume integral: flux_ranocha (:366-395) plus half
  // the nonconservative flux_nonconservative_waruszewski_etal (:186-205), both
  // with the averaged contravariant vector (n1, n2).  Returns Fa = F + G/2 (to
  // node a, weighted by Dsplit[a,b]) and Fb = F - G/2 (to node b, Dsplit[b,a]);
  // G(b,a) = -G(a,b).  p_ll p_rr inv_ln_mean(rho_ll p_rr, rho_rr p_ll) is
  // evaluated as the equal inv_ln_mean(rho_ll/p_ll, rho_rr/p_rr), the mean of
  // the reciprocals of the node values p/rho.  With g = (phi_b - phi_a) / 4 the
  // momentum fluxes of the two sides are f1 v + n (p_avg +- 2 rho_mean g), and
  // half the energy fluxes
  //   f1 (v_a.v_b / 4 + mean(p/rho) / (2 (gamma - 1)) +- g) + (p_a vn_b + p_b vn_a) / 4.
  // Elements in range take fx_energy_pair (fixed_flux.cuh) instead.
  TAG_HD static void volume_pair(const Params& P, const double* qa, const double* qb,
                                 double n1, double n2, double* Fa, double* Fb) {
    const double R = ln_factor(qa[0], qb[0], log_difference(qa[6], qb[6]));
    const double Q = inv_ln_factor(qa[5], qb[5], log_difference(qa[7], qb[7]));
    const double rho_mean = (qa[0] + qb[0]) * R;
    const double v1 = qa[1] + qb[1], v2 = qa[2] + qb[2];
    // halved normal velocities of both nodes
    const double vna = fma(qa[2], n2, qa[1] * n1);
    const double vnb = fma(qb[2], n2, qb[1] * n1);
    const double f1 = rho_mean * (vna + vnb);
    const double g = qb[4] - qa[4];
    const double p_avg = qa[3] + qb[3], r2 = twice(rho_mean);
    const double pp = fma(r2, g, p_avg), pm = fma(-r2, g, p_avg);
    const double t1 = f1 * v1, t2 = f1 * v2;
    Fa[0] = f1;
    Fb[0] = f1;
    Fa[1] = fma(n1, pp, t1);
    Fb[1] = fma(n1, pm, t1);
    Fa[2] = fma(n2, pp, t2);
    Fb[2] = fma(n2, pm, t2);
    const double vv = fma(qa[2], qb[2], qa[1] * qb[1]);
    const double x = fma(qa[5] + qb[5], Q, vv);
    const double e = fma(f1, x, fma(qa[3], vnb, qb[3] * vna));
    Fa[3] = fma(f1, g, e);
    Fb[3] = fma(-f1, g, e);
  }

  TAG_HD static void fixed_pair(const Params&, const double* qa, const double* qb,
                                const double* na, const double* nb, u64 Q, const FxShift& k,
                                i64* Fa, i64* Fb) {
    fx_energy_pair<2>(reinterpret_cast<const i64*>(qa), reinterpret_cast<const i64*>(qb),
                      reinterpret_cast<const i64*>(na), reinterpret_cast<const i64*>(nb), Q, k, Fa,
                      Fb);
  }

  // FluxLMARS (:397-430) between states ul, ur for the (unnormalised) normal n:
  //   p = (p_ll + p_rr)/2 - c rho (v_rr - v_ll) / (2 |n|),
  //   v = (v_ll + v_rr)/2 - (p_rr - p_ll) |n| / (2 c rho),  rho = (rho_ll + rho_rr)/2,
  // the reciprocals and the reciprocal root |n| on the integer pipe (the FP64
  // pipe bounds the interface kernel too), and p = (gamma - 1)(rho e -
  // |rho v|^2 / (2 rho)).
  TAG_DEV static void lmars(const Params& P, const double* ul, const double* ur, double n1,
                            double n2, double* F) {
    const double rho_ll = ul[0], rho_rr = ur[0];
    const double srho = rho_ll + rho_rr;
    const double irl = int_rcp(rho_ll), irr = int_rcp(rho_rr), isum = int_rcp(srho);
    const double p_ll = P.gm1 * fma(-0.5 * irl, fma(ul[2], ul[2], ul[1] * ul[1]), ul[3]);
    const double p_rr = P.gm1 * fma(-0.5 * irr, fma(ur[2], ur[2], ur[1] * ur[1]), ur[3]);
    const double v_ll = fma(ul[2], n2, ul[1] * n1) * irl;
    const double v_rr = fma(ur[2], n2, ur[1] * n1) * irr;
    const double nsq = fma(n2, n2, n1 * n1);
    const double inorm = int_rsqrt(nsq), norm_ = nsq * inorm;
    const double p = 0.5 * (p_ll + p_rr) - P.quarter_c * srho * (v_rr - v_ll) * inorm;
    const double v = 0.5 * (v_ll + v_rr) - P.inv_c * (p_rr - p_ll) * norm_ * isum;
    if (v >= 0.0) {
      F[0] = ul[0] * v; F[1] = ul[1] * v; F[2] = ul[2] * v; F[3] = ul[3] * v + p_ll * v;
    } else {
      F[0] = ur[0] * v; F[1] = ur[1] * v; F[2] = ur[2] * v; F[3] = ur[3] * v + p_rr * v;
    }
    F[1] += p * n1;
    F[2] += p * n2;
  }

  // Interface: surface flux (FluxLMARS, flux_zero) with the primary's outward
  // normal; F is stored for the primary and -F for the secondary.
  TAG_DEV static void surface_flux(const Params& P, const double* ul, const double* ur, double n1,
                                   double n2, double* F) {
    lmars(P, ul, ur, n1, n2, F);
  }

  // Slip wall.  kind TAG_BC_SLIP_WALL_STRUCTURED: normal (n1, n2) is the
  // sign-corrected contravariant vector in the +xi/+eta sense; the reference
  // method :102-129 mirrors v2 and orders the states by the parity of the face;
  // the returned flux is OUTWARD (negated on xi-/eta- faces).
  // kind TAG_BC_SLIP_WALL_NORMAL: (n1, n2) is the outward normal; :77-100.
  TAG_DEV static void boundary_flux(const Params& P, const double* ui, double n1, double n2,
                                    int face, int kind, double* F) {
    if (kind == TAG_BC_SLIP_WALL_STRUCTURED) {
      const double ub[5] = {ui[0], ui[1], -ui[2], ui[3], ui[4]};
      if (face & 1) {
        lmars(P, ui, ub, n1, n2, F);
      } else {
        lmars(P, ub, ui, n1, n2, F);
        F[0] = -F[0]; F[1] = -F[1]; F[2] = -F[2]; F[3] = -F[3];
      }
    } else {
      const double inn = int_rsqrt(fma(n2, n2, n1 * n1));
      const double nx = n1 * inn, ny = n2 * inn;
      const double un = nx * ui[1] + ny * ui[2];
      const double ub[5] = {ui[0], ui[1] - 2.0 * un * nx, ui[2] - 2.0 * un * ny, ui[3], ui[4]};
      lmars(P, ui, ub, n1, n2, F);
    }
  }

  // max_abs_speeds (:518-524)
  TAG_DEV static void max_speeds(const Params& P, const double* u, double& l1, double& l2) {
    const double irho = int_rcp(u[0]);
    const double v1 = u[1] * irho, v2 = u[2] * irho;
    const double p = P.gm1 * (u[3] - 0.5 * (u[1] * v1 + u[2] * v2));
    const double c = int_sqrt(P.gamma * p * irho);
    l1 = fabs(v1) + c;
    l2 = fabs(v2) + c;
  }
};

}  // namespace tag
