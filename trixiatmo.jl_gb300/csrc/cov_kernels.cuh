// Covariant shallow-water equations on a 2D manifold (the cubed sphere):
// device physics and kernels.
//
// Reference: src/equations/covariant_shallow_water.jl (fluxes :155-176,
// sources :216-243, speeds :246-305), covariant_shallow_water_split.jl
// (flux_ec :101-116, nonconservative fluxes :142-220, sources :273-302), the
// Lax-Friedrichs dissipation of src/equations/equations.jl:243-257, and the
// covariant DGSEM of src/solvers/dgsem_p4est/dg_2d_manifold_in_3d_covariant.jl
// (weak form :98-131, flux differencing :135-234, interfaces :239-432,
// sources :435-452, apply_jacobian :461-478), max_dt of
// src/callbacks_step/stepsize_dg2d.jl:47-71.
//
// A handle holds one or more element groups; a group is a run of elements of
// one polynomial degree (an uneven ensemble has one group per run of members
// with equal degree).  Every stage is one interface launch and one element
// launch over all groups: each CTA finds its group and runs the body
// instantiated for that group's n.  The solution is u[node][3] with the
// nodes of each element contiguous; aux[node][26] is the reference's
// aux_node_vars; pk[node][16] a packed copy of what the element kernel reads.
#pragma once
#include "cov_params.cuh"
#include "dg2d_kernels.cuh"

namespace tag {

// packed per-node element data: area element, contravariant metric, covariant
// metric (standard form: the first two are the contractions Gamma^i : G_con of
// the pressure source), bottom topography, the geometric source's coefficients
// of hv^1 v^1, hv^1 v^2 and hv^2 v^2 in both components, f J and 1/J
enum CovPack : int {
  kPJ = 0, kPGc11, kPGc12, kPGc22, kPGv11, kPGv12, kPGv22, kPHs,
  kPS100, kPS101, kPS111, kPS200, kPS201, kPS211, kPFJ, kPInvJ, kPack = 16
};

TAG_DEV int cov_find_group(const CovGroups& G, int blk, bool iface) {
  int lo = 0;
  for (int k = 1; k < G.count; ++k)
    if ((iface ? G.g[k].iblk0 : G.g[k].blk0) <= blk) lo = k;
  return lo;
}

// packs aux (26), the Coriolis parameter f = 2 Omega z / |x| times J and 1/J per
// node.  The geometric source is a contraction of hv (x) v with geometry alone:
//   standard: Gamma^i : (hv (x) v + g h^2/2 G_con);
//   split: (Gamma^i : T - G_con^ij w_j) / 2 with w_j = Gamma^k_jl (G_cov T)_kl,
// so its six coefficients are formed here, once, instead of 60 operations per
// node and stage.
__global__ void k_cov_pack(const double* __restrict__ aux, const double* __restrict__ xyz,
                           long nodes, double omega, int split, double* __restrict__ pk) {
  const long q = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nodes) return;
  const double* a = aux + q * 26;
  double* p = pk + q * kPack;
  const double J = a[12], v11 = a[13], v12 = a[14], v22 = a[15];
  const double c11 = a[16], c12 = a[17], c22 = a[18];
  const double g111 = a[20], g112 = a[21], g122 = a[22], g211 = a[23], g212 = a[24], g222 = a[25];
  p[kPJ] = J;
  p[kPGc11] = c11; p[kPGc12] = c12; p[kPGc22] = c22;
  p[kPGv11] = v11; p[kPGv12] = v12; p[kPGv22] = v22;
  p[kPHs] = a[19];
  // symmetric parts Gamma^i : T
  double s1[3] = {g111, 2.0 * g112, g122}, s2[3] = {g211, 2.0 * g212, g222};
  if (split) {
    const double w1[3] = {g111 * v11 + g211 * v12,
                          (g111 * v12 + g112 * v11) + (g211 * v22 + g212 * v12),
                          g112 * v12 + g212 * v22};
    const double w2[3] = {g112 * v11 + g212 * v12,
                          (g112 * v12 + g122 * v11) + (g212 * v22 + g222 * v12),
                          g122 * v12 + g222 * v22};
    for (int k = 0; k < 3; ++k) {
      s1[k] = 0.5 * (s1[k] - (c11 * w1[k] + c12 * w2[k]));
      s2[k] = 0.5 * (s2[k] - (c12 * w1[k] + c22 * w2[k]));
    }
  } else {
    p[kPGv11] = g111 * c11 + 2.0 * g112 * c12 + g122 * c22;
    p[kPGv12] = g211 * c11 + 2.0 * g212 * c12 + g222 * c22;
  }
  for (int k = 0; k < 3; ++k) {
    p[kPS100 + k] = s1[k];
    p[kPS200 + k] = s2[k];
  }
  const double* x = xyz + q * 3;
  p[kPFJ] = 2.0 * omega * x[2] / sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]) * J;
  p[kPInvJ] = 1.0 / J;
}

// ---- pointwise physics on packed data -----------------------------------------
// contravariant fluxes of one node (standard or split form) in both directions,
// F[0..2] and F[3..5]: the momentum part is the symmetric J (hv (x) v), plus
// J G_con g h^2/2 in the standard form; ih = 1/h
TAG_DEV void cov_flux(const CovParams& P, const double* u, double ih, const double* p, double* F) {
  const double m1 = p[kPJ] * u[1], m2 = p[kPJ] * u[2];
  const double v1 = u[1] * ih, v2 = u[2] * ih;
  double T11 = m1 * v1, T12 = m1 * v2, T22 = m2 * v2;
  if (!P.split) {
    const double gt = p[kPJ] * (0.5 * P.g * u[0] * u[0]);
    T11 = fma(p[kPGc11], gt, T11);
    T12 = fma(p[kPGc12], gt, T12);
    T22 = fma(p[kPGc22], gt, T22);
  }
  F[0] = m1;
  F[1] = T11;
  F[2] = T12;
  F[3] = m2;
  F[4] = T12;
  F[5] = T22;
}

// source_terms_geometric_coriolis (standard or split), after apply_jacobian,
// from the coefficients of k_cov_pack
TAG_DEV void cov_source(const CovParams& P, const double* u, double ih, const double* p,
                        double* s) {
  const double hv0 = u[1], hv1 = u[2];
  const double v0 = hv0 * ih, v1 = hv1 * ih;
  const double T00 = hv0 * v0, T01 = hv0 * v1, T11 = hv1 * v1;
  double sg0 = fma(p[kPS111], T11, fma(p[kPS101], T01, p[kPS100] * T00));
  double sg1 = fma(p[kPS211], T11, fma(p[kPS201], T01, p[kPS200] * T00));
  if (!P.split) {
    const double gt = 0.5 * P.g * u[0] * u[0];
    sg0 = fma(gt, p[kPGv11], sg0);
    sg1 = fma(gt, p[kPGv12], sg1);
  }
  const double f0 = p[kPFJ] * hv0, f1 = p[kPFJ] * hv1;
  s[0] = 0.0;
  s[1] = -fma(p[kPGc12], f0, fma(-p[kPGc11], f1, sg0));
  s[2] = -fma(p[kPGc22], f0, fma(-p[kPGc12], f1, sg1));
}

// ---- interface fluxes ------------------------------------------------------------
// Geometry of the two sides of an interface node, packed once per handle from
// the reference's aux layout (A column-major at 0..5, the contravariant basis
// column-major at 6..11, J at 12, G_11 G_12 G_22 at 13..15, G^11 G^12 G^22 at
// 16..18) for the face normal o of the side:
//   M: the other side's (hv^1, hv^2) in this side's basis, row-major;
//   J with the face's outward sign, G^{1o}, G^{2o}, sqrt(g G^{oo});
//   E = G_con G_cov - 1 (rounding of the stored metric), row-major.
// In place of 19 numbers of either node: 76 instead of 160 FP64 operations per
// interface node (the FP64 pipe is the bound).  Arrays of kIfSide values per side, the
// interface nodes contiguous, so a warp's loads are coalesced.
enum CovIfPack : int {
  kIM = 0, kIJ = 4, kIG1, kIG2, kISpeed, kIE = 8, kIfSide = 12, kIfPack = 2 * kIfSide
};

struct CovIfNode {
  int e0, e1, f0, f1, l1;
  long q0, q1;  // nodes of the two sides
};
TAG_DEV CovIfNode cov_if_node(const CovGroup& G, int n, int k, int l,
                              const int* __restrict__ if_e, const int* __restrict__ if_f,
                              const int* __restrict__ if_flip) {
  CovIfNode r;
  const int kk = G.if0 + k;
  r.e0 = if_e[2 * kk];
  r.e1 = if_e[2 * kk + 1];
  r.f0 = if_f[2 * kk];
  r.f1 = if_f[2 * kk + 1];
  r.l1 = if_flip[kk] ? n - 1 - l : l;
  int i0, j0, i1, j1;
  face_node(r.f0, l, n, i0, j0);
  face_node(r.f1, r.l1, n, i1, j1);
  r.q0 = G.node0 + (long)(r.e0 - G.e0) * n * n + j0 * n + i0;
  r.q1 = G.node0 + (long)(r.e1 - G.e0) * n * n + j1 * n + i1;
  return r;
}

// one side: `mine` and `other` aux rows, face f of `mine`
TAG_DEV void cov_pack_side(const double* mine, const double* other, int f, double g,
                           double* __restrict__ p, long stride) {
  const int o = f >> 1;
  for (int r = 0; r < 2; ++r)
    for (int c = 0; c < 2; ++c)
      p[(kIM + 2 * r + c) * stride] = mine[6 + r] * other[3 * c] + mine[8 + r] * other[3 * c + 1] +
                                      mine[10 + r] * other[3 * c + 2];
  const double v11 = mine[13], v12 = mine[14], v22 = mine[15];
  const double c11 = mine[16], c12 = mine[17], c22 = mine[18];
  p[kIJ * stride] = f & 1 ? mine[12] : -mine[12];
  p[kIG1 * stride] = o ? c12 : c11;
  p[kIG2 * stride] = o ? c22 : c12;
  p[kISpeed * stride] = sqrt(g * (o ? c22 : c11));
  p[(kIE + 0) * stride] = fma(c11, v11, fma(c12, v12, -1.0));
  p[(kIE + 1) * stride] = fma(c11, v12, c12 * v22);
  p[(kIE + 2) * stride] = fma(c12, v11, c22 * v12);
  p[(kIE + 3) * stride] = fma(c12, v12, fma(c22, v22, -1.0));
}

// grid as k_cov_interface
__global__ void k_cov_pack_interfaces(double g, const CovGroups* __restrict__ GG,
                                      const double* __restrict__ aux,
                                      const int* __restrict__ if_e, const int* __restrict__ if_f,
                                      const int* __restrict__ if_flip, long nodes,
                                      double* __restrict__ ipk) {
  const CovGroup& G = GG->g[cov_find_group(*GG, blockIdx.x, true)];
  const int t = (blockIdx.x - G.iblk0) * blockDim.x + threadIdx.x;
  const int n = G.n;
  if (t >= G.nif * n) return;
  const CovIfNode r = cov_if_node(G, n, t / n, t % n, if_e, if_f, if_flip);
  double* p = ipk + G.ifnode0 + t;
  cov_pack_side(aux + r.q0 * 26, aux + r.q1 * 26, r.f0, g, p, nodes);
  cov_pack_side(aux + r.q1 * 26, aux + r.q0 * 26, r.f1, g, p + kIfSide * nodes, nodes);
}

// Outward surface flux (+ 0.5 nonconservative) of one side, face f, in its own
// basis and with its own geometry p[kIfSide] for both states (the reference
// passes aux_vars_ll twice).  mine, w: this side's state and the other's in this
// side's basis; their reciprocals and square roots of h; hph = g h h' / 2.
TAG_DEV void cov_side_flux(const CovParams& P, const double* mine, const double* w, double ihm,
                           double ihw, double sqm, double sqw, double hph, int f,
                           const double* p, double* F) {
  const bool second = f >> 1, plus = f & 1;
  // a: left state, c: right state along the face's direction
  const double a0 = plus ? mine[0] : w[0], c0 = plus ? w[0] : mine[0];
  const double a1 = plus ? mine[1] : w[1], c1 = plus ? w[1] : mine[1];
  const double a2 = plus ? mine[2] : w[2], c2 = plus ? w[2] : mine[2];
  const double iha = plus ? ihm : ihw, ihc = plus ? ihw : ihm;
  const double va1 = a1 * iha, va2 = a2 * iha, vc1 = c1 * ihc, vc2 = c2 * ihc;
  const double ao = second ? a2 : a1, co = second ? c2 : c1;
  const double vao = second ? va2 : va1, vco = second ? vc2 : vc1;
  const double g1 = p[kIG1], g2 = p[kIG2];
  double F0 = 0.5 * (ao + co), F1, F2;
  if (P.surf_sym == 1) {
    const double hm = 0.5 * F0;
    F1 = (va1 + vc1) * hm;
    F2 = (va2 + vc2) * hm;
  } else {
    F1 = 0.5 * fma(ao, va1, co * vc1);
    F2 = 0.5 * fma(ao, va2, co * vc2);
    if (!P.split) {
      const double gt = 0.25 * P.g * fma(a0, a0, c0 * c0);
      F1 = fma(g1, gt, F1);
      F2 = fma(g2, gt, F2);
    }
  }
  if (P.surf_diss) {
    const double s = -0.5 * fmax(fma(plus ? sqm : sqw, p[kISpeed], fabs(vao)),
                                 fma(plus ? sqw : sqm, p[kISpeed], fabs(vco)));
    F0 = fma(s, c0 - a0, F0);
    F1 = fma(s, c1 - a1, F1);
    F2 = fma(s, c2 - a2, F2);
  }
  if (P.surf_nc) {
    F1 = fma(g1, hph, F1);
    F2 = fma(g2, hph, F2);
    if (P.surf_nc == 1) {
      // flux_nonconservative_ec with one geometry (no topography jump): the
      // velocity term is hv_a^o / 2 (G_con G_cov - 1) v_c
      const double q = 0.25 * ao;
      F1 = fma(q, fma(p[kIE], vc1, p[kIE + 1] * vc2), F1);
      F2 = fma(q, fma(p[kIE + 2], vc1, p[kIE + 3] * vc2), F2);
    }
  }
  const double J = p[kIJ];
  F[0] = J * F0;
  F[1] = J * F1;
  F[2] = J * F2;
}

template <int n>
TAG_DEV void cov_interface_body(const CovParams& P, const CovGroup& G, int lblk,
                                const double* u, const double* __restrict__ ipk, long nodes,
                                const int* __restrict__ if_e, const int* __restrict__ if_f,
                                const int* __restrict__ if_flip, double* __restrict__ sfv) {
  const int t = lblk * blockDim.x + threadIdx.x;
  const int k = t / n, l = t % n;
  if (k >= G.nif) return;
  double p[kIfPack];
#pragma unroll
  for (int j = 0; j < kIfPack; ++j)
    p[j] = (j % kIfSide < kIE || P.surf_nc == 1) ? __ldg(ipk + j * nodes + G.ifnode0 + t) : 0.0;
  const CovIfNode r = cov_if_node(G, n, k, l, if_e, if_f, if_flip);
  double ul[3], ur[3], rt[3], lt[3], Fl[3], Fr[3];
  wait_for_previous();
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    ul[v] = u[r.q0 * 3 + v];
    ur[v] = u[r.q1 * 3 + v];
  }
  const double* pr = p + kIfSide;
  rt[0] = ur[0];
  rt[1] = fma(p[kIM], ur[1], p[kIM + 1] * ur[2]);
  rt[2] = fma(p[kIM + 2], ur[1], p[kIM + 3] * ur[2]);
  lt[0] = ul[0];
  lt[1] = fma(pr[kIM], ul[1], pr[kIM + 1] * ul[2]);
  lt[2] = fma(pr[kIM + 2], ul[1], pr[kIM + 3] * ul[2]);
  const double ihl = int_rcp(ul[0]), ihr = int_rcp(ur[0]);
  const double sql = P.surf_diss ? int_sqrt(ul[0]) : 0.0;
  const double sqr = P.surf_diss ? int_sqrt(ur[0]) : 0.0;
  const double hph = P.surf_nc ? 0.5 * P.g * ul[0] * ur[0] : 0.0;
  cov_side_flux(P, ul, rt, ihl, ihr, sql, sqr, hph, r.f0, p, Fl);
  cov_side_flux(P, ur, lt, ihr, ihl, sqr, sql, hph, r.f1, pr, Fr);
  release_next();
  double* s0 = sfv + G.sf0 + ((long)(r.e0 - G.e0) * 4 + r.f0) * n * 3 + l * 3;
  double* s1 = sfv + G.sf0 + ((long)(r.e1 - G.e0) * 4 + r.f1) * n * 3 + r.l1 * 3;
#pragma unroll
  for (int v = 0; v < 3; ++v) {
    s0[v] = Fl[v];
    s1[v] = Fr[v];
  }
}

// 128-thread CTAs (the interface node counts fill the SMs evenly: 43,200 nodes
// are 169 CTAs of 256 on 152 SMs)
constexpr int kCovIfThreads = 128;
__global__ void __launch_bounds__(kCovIfThreads)
    k_cov_interface(CovParams P, const CovGroups* __restrict__ GG, const double* u,
                    const double* __restrict__ ipk, long nodes, const int* __restrict__ if_e,
                    const int* __restrict__ if_f, const int* __restrict__ if_flip,
                    double* __restrict__ sfv) {
  const int gi = cov_find_group(*GG, blockIdx.x, true);
  const CovGroup& G = GG->g[gi];
  const int lblk = blockIdx.x - G.iblk0;
  switch (G.n) {
    case 4: cov_interface_body<4>(P, G, lblk, u, ipk, nodes, if_e, if_f, if_flip, sfv); break;
    case 6: cov_interface_body<6>(P, G, lblk, u, ipk, nodes, if_e, if_f, if_flip, sfv); break;
    case 8: cov_interface_body<8>(P, G, lblk, u, ipk, nodes, if_e, if_f, if_flip, sfv); break;
    case 2: cov_interface_body<2>(P, G, lblk, u, ipk, nodes, if_e, if_f, if_flip, sfv); break;
    case 3: cov_interface_body<3>(P, G, lblk, u, ipk, nodes, if_e, if_f, if_flip, sfv); break;
    case 5: cov_interface_body<5>(P, G, lblk, u, ipk, nodes, if_e, if_f, if_flip, sfv); break;
    case 7: cov_interface_body<7>(P, G, lblk, u, ipk, nodes, if_e, if_f, if_flip, sfv); break;
    default: break;
  }
}

// ---- element kernel --------------------------------------------------------------
// One thread per node (epb n^2 of 128 or 256 threads).  Shared memory per node:
// flux differencing: v1, v2, (G_cov v)_1, (G_cov v)_2, J hv^1, J hv^2, h, h_s, J,
// G^11, G^12, G^22, g h^2 / 2 (13 doubles, an odd stride); weak form: the two
// contravariant fluxes.
constexpr int kCovQ = 13;
__host__ __device__ constexpr int cov_elem_doubles(int n) { return n * n * kCovQ; }

// VK: 0 weak form (VolumeIntegralWeakForm), 1 flux differencing; a template
// parameter so that each volume kind gets its own register allocation
template <int n, int MODE, int VK>
TAG_DEV void cov_element_body(const CovParams& P, const CovGroup& G, int lblk,
                              const BasisDev* __restrict__ bases, double* u,
                              double* __restrict__ du, double* __restrict__ kreg,
                              const double* __restrict__ pk, const double* sfv,
                              StageArgs st, double* smem, unsigned& bad) {
  constexpr int nn = n * n;
  BasisDev* sb = reinterpret_cast<BasisDev*>(smem);
  double* q = smem + sizeof(BasisDev) / sizeof(double);
  const int el_first = lblk * G.epb;
  const int ne = min(G.epb, G.ne - el_first);
  if (ne <= 0) return;
  for (int t = threadIdx.x; t < (int)(sizeof(BasisDev) / sizeof(double)); t += blockDim.x)
    smem[t] = reinterpret_cast<const double*>(bases + G.basis)[t];
  const int el = threadIdx.x / nn, node = threadIdx.x % nn;
  const bool act = el < ne;
  const int i = node % n, j = node / n;
  const long gq = G.node0 + (long)(el_first + el) * nn + node;
  double ui[3], ih = 0.0;  // ih = 1/h, shared by the fluxes and the source
  const bool regrouped = VK == 1 && P.split && P.vol_sym <= 1;
  double* qn = q + threadIdx.x * kCovQ;
  const double* __restrict__ pg = pk + gq * kPack;  // re-read where needed (L1 hit)
  if (act) {
    double p[kPack];
#pragma unroll
    for (int k = 0; k < kPack; ++k) p[k] = __ldg(pg + k);
    wait_for_previous();
#pragma unroll
    for (int v = 0; v < 3; ++v) ui[v] = u[gq * 3 + v];
    ih = int_rcp(ui[0]);
    if constexpr (VK == 0) {
      cov_flux(P, ui, ih, p, qn);
    } else {
      const double v1 = ui[1] * ih, v2 = ui[2] * ih;
      qn[0] = v1;
      qn[1] = v2;
      qn[2] = p[kPGv11] * v1 + p[kPGv12] * v2;
      qn[3] = p[kPGv12] * v1 + p[kPGv22] * v2;
      qn[4] = p[kPJ] * ui[1];
      qn[5] = p[kPJ] * ui[2];
      if (regrouped) {
        qn[6] = ui[0] + p[kPHs];
        qn[7] = v1 * qn[4];
        qn[8] = v2 * qn[4];
        qn[9] = v1 * qn[5];
        qn[10] = v2 * qn[5];
      } else {
        qn[6] = ui[0];
        qn[7] = p[kPHs];
        qn[8] = p[kPJ];
        qn[9] = p[kPGc11];
        qn[10] = p[kPGc12];
        qn[11] = p[kPGc22];
        qn[12] = 0.5 * P.g * ui[0] * ui[0];
      }
    }
  }
  __syncthreads();
  release_next();
  double un[3] = {0.0, 0.0, 0.0};
  if (act) {
    const double* eq = q + el * nn * kCovQ;
    double acc[3] = {0.0, 0.0, 0.0};
    if constexpr (VK == 0) {
#pragma unroll
      for (int b = 0; b < n; ++b) {
        const double d1 = sb->Dh[i * n + b], d2 = sb->Dh[j * n + b];
        const double* F1 = eq + (j * n + b) * kCovQ;
        const double* F2 = eq + (b * n + i) * kCovQ + 3;
#pragma unroll
        for (int v = 0; v < 3; ++v) acc[v] = fma(d2, F2[v], fma(d1, F1[v], acc[v]));
      }
    } else if (regrouped) {
      // Split form with flux_central or flux_ec (and flux_nonconservative_ec):
      // every pair flux is a sum of products of a node-a factor and a node-b
      // factor, so each line sum sum_b D_ab f(a, b) is formed from contractions
      // sum_b D_ab x_b of node-b quantities (the pair terms of
      // covariant_shallow_water_split.jl:100-215 regrouped; with the products
      // v J hv formed per node, eight multiply-adds per partner node).  b = a is
      // left out of the symmetric part and kept in the nonconservative part, as
      // in the pairwise form.
      const double* qa = qn;
      const double gh = P.g * ui[0];
      const double gc11 = __ldg(pg + kPGc11), gc12 = __ldg(pg + kPGc12),
                   gc22 = __ldg(pg + kPGc22), hs_a = __ldg(pg + kPHs);
      double nc1 = 0.0, nc2 = 0.0;
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        const double hvo_a = d ? ui[2] : ui[1];
        const double Jhvo_a = d ? qa[5] : qa[4];
        const int a = d ? j : i;
        double A1 = 0.0, A2 = 0.0, A3 = 0.0, A4 = 0.0, A5 = 0.0;
        double B2 = 0.0, B3 = 0.0, BH = 0.0;
#pragma unroll
        for (int b = 0; b < n; ++b) {
          const double* qb = eq + (d ? b * n + i : j * n + b) * kCovQ;
          const double Dab = sb->Ds[a * n + b];
          if (b != a) {
            A1 = fma(Dab, qb[4 + d], A1);
            A2 = fma(Dab, qb[0], A2);
            A3 = fma(Dab, qb[7 + 2 * d], A3);
            A4 = fma(Dab, qb[1], A4);
            A5 = fma(Dab, qb[8 + 2 * d], A5);
          }
          if (P.vol_nc) {
            B2 = fma(Dab, qb[2], B2);
            B3 = fma(Dab, qb[3], B3);
            BH = fma(Dab, qb[6], BH);
          }
        }
        const double SD = sb->Dsum[a];  // the row of D_split without b = a
        const double m = fma(Jhvo_a, SD, A1);
        acc[0] = fma(0.5, m, acc[0]);
        if (P.vol_sym == 1) {
          // flux_ec: f = m (1, (v_a + v_b) / 2), m = (J hv_a + J hv_b) / 2
          acc[1] = fma(0.25, fma(qa[0], m, fma(Jhvo_a, A2, A3)), acc[1]);
          acc[2] = fma(0.25, fma(qa[1], m, fma(Jhvo_a, A4, A5)), acc[2]);
        } else {
          // flux_central of the split fluxes: (J hv v_a + J hv v_b) / 2
          acc[1] = fma(0.5, fma(qa[7 + 2 * d], SD, A3), acc[1]);
          acc[2] = fma(0.5, fma(qa[8 + 2 * d], SD, A5), acc[2]);
        }
        if (P.vol_nc) {
          const double Daa = sb->Ds[a * n + a];
          const double B0 = fma(Daa, qa[0], A2), B1 = fma(Daa, qa[1], A4);
          const double half_m = 0.5 * hvo_a;
          const double ph = gh * fma(-hs_a, SD + Daa, BH);
          nc1 = fma(d ? gc12 : gc11, ph, fma(half_m, fma(gc11, B2, fma(gc12, B3, -B0)), nc1));
          nc2 = fma(d ? gc22 : gc12, ph, fma(half_m, fma(gc12, B2, fma(gc22, B3, -B1)), nc2));
        }
      }
      const double hJ = 0.5 * __ldg(pg + kPJ);
      acc[1] = fma(hJ, nc1, acc[1]);
      acc[2] = fma(hJ, nc2, acc[2]);
    } else {
      const double* qa = qn;
      const double h_a = ui[0], hs_a = qa[7], J_a = qa[8];
      double nc1 = 0.0, nc2 = 0.0;
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        const double hvo_a = d ? ui[2] : ui[1];
        const double Jhvo_a = d ? qa[5] : qa[4];
        const double gco0 = d ? qa[10] : qa[9], gco1 = d ? qa[11] : qa[10];
        const int a = d ? j : i;
#pragma unroll
        for (int b = 0; b < n; ++b) {
          const double* qb = eq + (d ? b * n + i : j * n + b) * kCovQ;
          const double Dab = sb->Ds[a * n + b];
          if (b != a) {
            const double Jhvo_b = d ? qb[5] : qb[4];
            double f0, f1, f2;
            if (P.vol_sym == 1) {
              const double m = 0.5 * (Jhvo_a + Jhvo_b);
              f0 = m;
              f1 = 0.5 * (qa[0] + qb[0]) * m;
              f2 = 0.5 * (qa[1] + qb[1]) * m;
            } else if (P.split) {
              f0 = 0.5 * (Jhvo_a + Jhvo_b);
              f1 = 0.5 * (Jhvo_a * qa[0] + Jhvo_b * qb[0]);
              f2 = 0.5 * (Jhvo_a * qa[1] + Jhvo_b * qb[1]);
            } else {
              const double gb0 = d ? qb[10] : qb[9], gb1 = d ? qb[11] : qb[10];
              f0 = 0.5 * (Jhvo_a + Jhvo_b);
              f1 = 0.5 * ((Jhvo_a * qa[0] + J_a * gco0 * qa[12]) + (Jhvo_b * qb[0] + qb[8] * gb0 * qb[12]));
              f2 = 0.5 * ((Jhvo_a * qa[1] + J_a * gco1 * qa[12]) + (Jhvo_b * qb[1] + qb[8] * gb1 * qb[12]));
            }
            acc[0] = fma(Dab, f0, acc[0]);
            acc[1] = fma(Dab, f1, acc[1]);
            acc[2] = fma(Dab, f2, acc[2]);
          }
          if (P.vol_nc) {
            const double half_m = 0.5 * hvo_a;
            const double ph = P.g * h_a * (qb[6] + (qb[7] - hs_a));
            const double g0 = J_a * (half_m * (qa[9] * qb[2] + qa[10] * qb[3] - qb[0]) + gco0 * ph);
            const double g1 = J_a * (half_m * (qa[10] * qb[2] + qa[11] * qb[3] - qb[1]) + gco1 * ph);
            nc1 = fma(Dab, g0, nc1);
            nc2 = fma(Dab, g1, nc2);
          }
        }
      }
      acc[1] += 0.5 * nc1;
      acc[2] += 0.5 * nc2;
    }
    const double* se = sfv + G.sf0 + (long)(el_first + el) * 4 * n * 3;
    // one multiply-add per direction (a node lies on at most one of its faces)
    if (i == 0 || i == n - 1) {
      const double w = i == 0 ? sb->winv0 : sb->winvN;
#pragma unroll
      for (int v = 0; v < 3; ++v) acc[v] = fma(se[((i == 0 ? 0 : 1) * n + j) * 3 + v], w, acc[v]);
    }
    if (j == 0 || j == n - 1) {
      const double w = j == 0 ? sb->winv0 : sb->winvN;
#pragma unroll
      for (int v = 0; v < 3; ++v) acc[v] = fma(se[((j == 0 ? 2 : 3) * n + i) * 3 + v], w, acc[v]);
    }
    double s[3];
    {
      double p[kPack];
#pragma unroll
      for (int k = 0; k < kPack; ++k) p[k] = __ldg(pg + k);
      cov_source(P, ui, ih, p, s);
    }
    const double fac = -__ldg(pg + kPInvJ);
    const int e = G.e0 + el_first + el;
    double dv[3];
#pragma unroll
    for (int v = 0; v < 3; ++v) {
      dv[v] = acc[v] * fac + s[v];
      if (not_finite(dv[v])) bad |= TAG_S_NAN;
    }
    if (not_positive(ui[0])) bad |= TAG_S_NEG_DENSITY;
    if (MODE == kModeRhs) {
#pragma unroll
      for (int v = 0; v < 3; ++v) du[gq * 3 + v] = dv[v];
    } else {
      const double dt = st.dt[st.member ? st.member[e] : 0];
#pragma unroll
      for (int v = 0; v < 3; ++v) {
        un[v] = stage_value(st, ui[v], kreg + gq * 3 + v, dt, dv[v]);
        u[gq * 3 + v] = un[v];
      }
    }
  }
  if (MODE == kModeStage && st.max_speed != nullptr) {
    // the step's result to the registered sink (host memory over the host
    // link).  A warp's nodes are consecutive, so its 32 nodes x 3 values are
    // 96 consecutive doubles: lane l stores doubles l, l + 32 and l + 64,
    // fetched from their nodes' lanes, so that every store is contiguous
    if (st.sink != nullptr) {
      const int lane = threadIdx.x & 31, w_first = threadIdx.x & ~31;
      const long q0 = G.node0 + (long)el_first * nn + w_first;
      const int valid = ne * nn - w_first;  // the warp's nodes in range (may be <= 0)
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const int d = lane + 32 * k, src = d / 3, c = d % 3;
        const double s0 = __shfl_sync(0xffffffffu, un[0], src);
        const double s1 = __shfl_sync(0xffffffffu, un[1], src);
        const double s2 = __shfl_sync(0xffffffffu, un[2], src);
        if (src < valid) st.sink[q0 * 3 + d] = c == 0 ? s0 : (c == 1 ? s1 : s2);
      }
    }
    // CFL speeds of the updated state, scaled by n: dt = cfl 2 / (n max_e(l1 + l2))
    __syncthreads();
    if (act) {
      const double ihn = int_rcp(un[0]);
      qn[0] = fabs(un[1] * ihn) + int_sqrt(__ldg(pg + kPGc11) * un[0] * P.g);
      qn[1] = fabs(un[2] * ihn) + int_sqrt(__ldg(pg + kPGc22) * un[0] * P.g);
    }
    // maxima over the rows, then over the element's rows
    __syncthreads();
    if (act && i == 0) {
      double m1 = 0.0, m2 = 0.0;
#pragma unroll
      for (int k = 0; k < n; ++k) {
        m1 = fmax(m1, qn[k * kCovQ]);
        m2 = fmax(m2, qn[k * kCovQ + 1]);
      }
      qn[2] = m1;
      qn[3] = m2;
    }
    __syncthreads();
    if (act && node == 0) {
      double m1 = 0.0, m2 = 0.0;
#pragma unroll
      for (int k = 0; k < n; ++k) {
        m1 = fmax(m1, qn[k * n * kCovQ + 2]);
        m2 = fmax(m2, qn[k * n * kCovQ + 3]);
      }
      const int e = G.e0 + el_first + el;
      atomic_max_nonneg(st.max_speed + (st.member ? st.member[e] : 0), n * (m1 + m2));
    }
  }
}

// At most 256 threads (128 on small meshes, chosen with the groups) and at least three
// CTAs per SM: up to 85 registers, which the
// FP64-latency-bound body uses for independent operations in flight
template <int MODE, int VK>
__global__ void __launch_bounds__(256, 3) k_cov_element(CovParams P, const CovGroups* __restrict__ GG,
                                                     const BasisDev* __restrict__ bases,
                                                     double* u, double* __restrict__ du,
                                                     double* __restrict__ kreg,
                                                     const double* __restrict__ pk,
                                                     const double* sfv, StageArgs st,
                                                     unsigned* __restrict__ status) {
  extern __shared__ double smem[];
  const int gi = cov_find_group(*GG, blockIdx.x, false);
  const CovGroup& G = GG->g[gi];
  const int lblk = blockIdx.x - G.blk0;
  unsigned bad = 0;
  switch (G.n) {
    case 4: cov_element_body<4, MODE, VK>(P, G, lblk, bases, u, du, kreg, pk, sfv, st, smem, bad); break;
    case 6: cov_element_body<6, MODE, VK>(P, G, lblk, bases, u, du, kreg, pk, sfv, st, smem, bad); break;
    case 8: cov_element_body<8, MODE, VK>(P, G, lblk, bases, u, du, kreg, pk, sfv, st, smem, bad); break;
    case 2: cov_element_body<2, MODE, VK>(P, G, lblk, bases, u, du, kreg, pk, sfv, st, smem, bad); break;
    case 3: cov_element_body<3, MODE, VK>(P, G, lblk, bases, u, du, kreg, pk, sfv, st, smem, bad); break;
    case 5: cov_element_body<5, MODE, VK>(P, G, lblk, bases, u, du, kreg, pk, sfv, st, smem, bad); break;
    case 7: cov_element_body<7, MODE, VK>(P, G, lblk, bases, u, du, kreg, pk, sfv, st, smem, bad); break;
    default: break;
  }
  if (bad) atomicOr(status, bad);
}

// scaled CFL speed n max_e(l1 + l2) of a host-set state, per member: one warp
// per element (blockDim a multiple of 32), the lanes stride over its nodes
__global__ void k_cov_max_speed(CovParams P, const CovGroups* __restrict__ GG,
                                const double* __restrict__ u, const double* __restrict__ pk,
                                const int* __restrict__ member, double* __restrict__ max_speed,
                                int nelem) {
  const int lane = threadIdx.x & 31;
  const int e = (int)(((long)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (e >= nelem) return;  // warp-uniform
  int gi = 0;
  for (int k = 1; k < GG->count; ++k)
    if (GG->g[k].e0 <= e) gi = k;
  const CovGroup& G = GG->g[gi];
  const int n = G.n, nn = n * n;
  const long q0 = G.node0 + (long)(e - G.e0) * nn;
  double m1 = 0.0, m2 = 0.0;
  for (int node = lane; node < nn; node += 32) {
    const double* uq = u + (q0 + node) * 3;
    const double* p = pk + (q0 + node) * kPack;
    const double ih = int_rcp(uq[0]);
    m1 = fmax(m1, fabs(uq[1] * ih) + int_sqrt(p[kPGc11] * uq[0] * P.g));
    m2 = fmax(m2, fabs(uq[2] * ih) + int_sqrt(p[kPGc22] * uq[0] * P.g));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    m1 = fmax(m1, __shfl_xor_sync(0xffffffffu, m1, o));
    m2 = fmax(m2, __shfl_xor_sync(0xffffffffu, m2, o));
  }
  if (lane == 0) atomic_max_nonneg(max_speed + (member ? member[e] : 0), n * (m1 + m2));
}

}  // namespace tag
