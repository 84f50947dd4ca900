"""Precision of the element-wide fixed-point volume integral (csrc/fixed_flux.cuh) on elements that are
flat, sheared or moving, against extended precision.

On the CPU the header is compiled for the host and one element's volume and surface integrals are
formed as the kernels form them, once in words and once in FP64, from the same node values.  Both carry
the rounding of the node values and of the operator, which is the larger part; the words' own rounding
is 2^-58 and less of the largest term.  So the words' error may not exceed FP64's; 1.25 leaves room for
the scatter of a root mean square over some thirty elements.  (With one scale for the components of a
contravariant vector the horizontal momentum was off by 3 at a width of 170 heights and by 320 at
20,000.)  A word that overflowed would be off by its whole scale: elements of random magnitudes are held
to 1e-9 of the largest term.

On the GPU an atmosphere at rest on flat meshes: the horizontal momentum is the derivative of the
pressure along horizontal lines and nothing else, each node's error below (n + 2) roundings of
p sum |D_split|: two of the node's pressure and its sum with the partner's, one of the product, n - 1 of
the sum (the operator is the one that the kernels get)."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_int_math import CSRC

HARNESS = r"""
#include <vector>
#include "phys_euler_energy_2d.cuh"
#include "phys_euler_energy_3d.cuh"
using namespace tag;
namespace tag { void set_last_error(const std::string&) {} }

// words[N][NA], fp64[N][NA]: sum over directions of the weighted pair fluxes and the end fluxes
// sf[2 D][N / n][NA] (outward) over the end weights; 1: the element is in range, 0: FP64 form
template <class Phys, int D>
int element(const double* par, int n, const double* Ds, const double* w, const double* u,
            const double* ja_in, const double* sf, double* words, double* fp64) {
  constexpr int NV = Phys::NV, NA = Phys::NA, NQ = Phys::NQ;
  const auto P = Phys::make_params(par);
  FxBasis b;
  load_fixed_basis(b, Ds, w, n);
  int stride[4] = {1, n, n * n, n * n * n};
  const int N = stride[D], face = N / n;
  std::vector<double> q(N * NQ), ja(ja_in, ja_in + N * D * D), acc(N * NA, 0.0);
  unsigned bad = 0;
  u32 mx[kMxCount] = {};
  const auto up = [&](int k, u32 v) { mx[k] = std::max(mx[k], v); };
  for (int i = 0; i < N; ++i) {
    double* p = &q[i * NQ];
    Phys::node_prims(P, u + i * NV, p, bad);
    p[D + 2] -= 0.25 * u[NV - 1];
    fx_node_maxima<D>(p, &ja[i * D * D], up);
  }
  const auto at = [&](int i, int d) { return i / stride[d] % n; };
  // node of end node k of face f
  const auto node = [&](int f, int k) {
    const int d = f / 2, low = k % stride[d], high = k / stride[d];
    return high * stride[d + 1] + (f & 1 ? n - 1 : 0) * stride[d] + low;
  };
  for (int f = 0; f < 2 * D; ++f)
    for (int k = 0; k < face * NA; ++k)
      up(fx_face_max<D>(k % NA, f / 2), high_magnitude(sf[f * face * NA + k]));
  FxScale<D> s;
  for (int d = 0; d < fx_groups(D); ++d) fx_scale<D>(mx, b, d, s);

  for (int d = 0; d < D; ++d)
    for (int i = 0; i < N; ++i)
      for (int m = at(i, d) + 1; m < n; ++m) {
        const int a = at(i, d), k = i + (m - a) * stride[d];
        double nrm[3], Fa[NA], Fb[NA];
        for (int c = 0; c < D; ++c) nrm[c] = ja[(i * D + d) * D + c] + ja[(k * D + d) * D + c];
        if constexpr (D == 2)
          Phys::volume_pair(P, &q[i * NQ], &q[k * NQ], nrm[0], nrm[1], Fa, Fb);
        else
          Phys::volume_pair(P, &q[i * NQ], &q[k * NQ], nrm, Fa, Fb);
        for (int v = 0; v < NA; ++v) {
          acc[i * NA + v] = std::fma(0.5 * Ds[a * n + m], Fa[v], acc[i * NA + v]);
          acc[k * NA + v] = std::fma(0.5 * Ds[m * n + a], Fb[v], acc[k * NA + v]);
        }
      }
  for (int f = 0; f < 2 * D; ++f)
    for (int k = 0; k < face; ++k)
      for (int v = 0; v < NA; ++v) {
        double& t = acc[node(f, k) * NA + v];
        const double iw = 1.0 / w[f & 1 ? n - 1 : 0];
        t = std::fma(sf[(f * face + k) * NA + v], v == NA - 1 ? 0.5 * iw : iw, t);
      }
  for (int i = 0; i < N * NA; ++i) fp64[i] = acc[i] * (i % NA == NA - 1 ? 2.0 : 1.0);
  if (!s.ok) return 0;

  std::vector<i64> A(D * N * NA, 0);
  for (int i = 0; i < N; ++i) {
    fx_convert_node<D>(&q[i * NQ], s);
    for (int k = 0; k < D * D; ++k)
      ja[i * D * D + k] = f64_from((u64)to_fixed(ja[i * D * D + k], s.sn[fx_group(D, k / D)][k % D] - 2));
  }
  for (int d = 0; d < D; ++d) {
    for (int i = 0; i < N; ++i)
      for (int m = at(i, d) + 1; m < n; ++m) {
        int a = i, c = i + (m - at(i, d)) * stride[d];
        const u64 Q = b.Q[at(i, d) * n + m];
        i64 Fa[NA], Fb[NA];
        if (Q & 1) std::swap(a, c);
        Phys::fixed_pair(P, &q[a * NQ], &q[c * NQ], &ja[(a * D + d) * D], &ja[(c * D + d) * D], Q,
                         s.k[fx_group(D, d)], Fa, Fb);
        for (int v = 0; v < NA; ++v) {
          A[(d * N + a) * NA + v] += Fa[v];
          A[(d * N + c) * NA + v] -= Fb[v];
        }
      }
    for (int e = 0; e < 2; ++e)
      for (int k = 0; k < face; ++k)
        for (int v = 0; v < NA; ++v)
          A[(d * N + node(2 * d + e, k)) * NA + v] +=
              fx_surface(sf[((2 * d + e) * face + k) * NA + v], s.sum[fx_group(D, d)][v] + (v == NA - 1), b.S[e]);
  }
  for (int i = 0; i < N; ++i)
    for (int v = 0; v < NA; ++v) {
      int pos[D], sd[D], scale;
      for (int d = 0; d < D; ++d) {
        pos[d] = at(i, d);
        sd[d] = s.sum[fx_group(D, d)][v];
      }
      const i64 t = fx_weighted_sum<D>(&A[i * NA + v], N * NA, b.W, pos, sd, scale);
      words[i * NA + v] =
          fx_zero(s, v) ? 0.0 : from_fixed(t, scale + b.kw) * (v == NA - 1 ? 2.0 : 1.0);
    }
  return 1;
}
extern "C" int run(int D, const double* par, int n, const double* Ds, const double* w, const double* u,
                   const double* ja, const double* sf, double* words, double* fp64) {
  return D == 2 ? element<PhysEnergy2D, 2>(par, n, Ds, w, u, ja, sf, words, fp64)
                : element<PhysEnergy3D, 3>(par, n, Ds, w, u, ja, sf, words, fp64);
}
"""
L = np.longdouble
CP, CV, G = 1004.0, 717.0, 9.81
GAMMA = L(CP) / L(CV)


@pytest.fixture(scope="module")
def host(tmp_path_factory, tg):
    d = tmp_path_factory.mktemp("fixed_flux")
    src, lib = d / "harness.cu", d / "harness.so"
    src.write_text(HARNESS)
    home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    nvcc = shutil.which("nvcc") or os.path.join(home, "bin", "nvcc")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-shared",
                    "-Xcompiler", "-fPIC", "-I", CSRC, str(src), "-o", str(lib)], check=True)
    fn = ctypes.CDLL(str(lib)).run
    dp = np.ctypeslib.ndpointer(np.float64, flags="C")
    fn.argtypes = [ctypes.c_int, dp, ctypes.c_int] + [dp] * 7
    basis = {n: tg.basis.LobattoLegendreBasis(n - 1) for n in range(2, 9)}

    def call(D, n, u, ja, sf):
        """(in words?, error of the words, of FP64, largest term), [nodes, variables]."""
        b = basis[n]
        Ds, w = np.ascontiguousarray(b.derivative_split), np.ascontiguousarray(b.weights)
        words, fp64 = np.zeros((n ** D, D + 2)), np.zeros((n ** D, D + 2))
        ok = fn(D, np.array([CP, CV, G, 340.0, 0, 0, 0, 0]), n, Ds, w, u, ja, sf, words, fp64)
        want, size = exact(D, n, u.astype(L), ja.astype(L), sf.astype(L))
        return ok, (words - want).astype(float), (fp64 - want).astype(float), size.astype(float)
    return call


def operator(n):
    """2 D - M^-1 B on Lobatto-Legendre nodes and the end weight, in extended precision."""
    def legendre(k, t):
        a, b = np.ones_like(t), t
        for j in range(1, k):
            a, b = b, ((2 * j + 1) * t * b - j * a) / (j + 1)
        return b if k else a
    m = n - 1
    x = np.array([-1.0] + sorted(np.polynomial.legendre.Legendre.basis(m).deriv().roots().real) + [1.0],
                 dtype=L)
    for _ in range(4):  # Newton on P_m' with P_m'' from Legendre's equation
        t = x[1:-1]
        dp = m * (legendre(m - 1, t) - t * legendre(m, t)) / (1 - t * t)
        x[1:-1] = t - dp * (1 - t * t) / (2 * t * dp - m * (m + 1) * legendre(m, t))
    c = np.array([np.prod([x[i] - x[j] for j in range(n) if j != i]) for i in range(n)], dtype=L)
    D = np.array([[c[i] / c[j] / (x[i] - x[j]) if i != j else L(0) for j in range(n)]
                  for i in range(n)], dtype=L)
    return 2 * D, L(2) / (n * (n - 1))  # (the diagonal is not used)


def ln_mean(x, y):
    t = (y - x) / (y + x)
    with np.errstate(invalid="ignore"):
        return (x + y) / 2 * np.where(t == 0, 1, t / np.arctanh(t))


def end_nodes(D, n, f):
    k, d = np.arange(n ** (D - 1)), f // 2
    return k // n ** d * n ** (d + 1) + (n - 1 if f & 1 else 0) * n ** d + k % n ** d


def exact(D, n, u, ja, sf, op=None):
    S, w0 = op or operator(n)
    rho, v, phi = u[:, 0], u[:, 1:1 + D] / u[:, :1], u[:, -1]
    p = (GAMMA - 1) * (u[:, 1 + D] - rho * (v * v).sum(1) / 2)
    N, i = n ** D, np.arange(n ** D)
    acc, size = np.zeros((N, D + 2), L), np.zeros((N, D + 2), L)
    for d in range(D):
        a = i // n ** d % n
        for b in range(n):
            k = i + (b - a) * n ** d
            nrm = (ja[:, d] + ja[k, d]) / 2
            va, vna, vnb = (v + v[k]) / 2, (v * nrm).sum(1), (v[k] * nrm).sum(1)
            f1 = ln_mean(rho, rho[k]) * (vna + vnb) / 2
            g = ln_mean(rho, rho[k]) * (phi[k] - phi) / 2
            e = 1 / ln_mean(rho / p, rho[k] / p[k]) / (GAMMA - 1)
            F = np.stack([f1, *(f1 * va[:, c] + ((p + p[k]) / 2 + g) * nrm[:, c] for c in range(D)),
                          f1 * ((v * v[k]).sum(1) / 2 + e) + (p * vnb + p[k] * vna) / 2 +
                          g * (vna + vnb) / 2], 1)
            F *= np.where(a == b, 0, S[a, b])[:, None]
            acc += F
            size = np.maximum(size, np.abs(F))
    for f in range(2 * D):
        acc[end_nodes(D, n, f)] += sf.reshape(2 * D, -1, D + 2)[f] / w0
    return acc, np.maximum(size, np.abs(acc))


def flat_element(D, n, width, wind, rng, tilt=0.0, scatter=0.0, height=1000.0, octaves=None):
    """Node values, contravariant vectors and the end fluxes of the element's own traces: `width`
    heights wide, hydrostatic, wind along it and 1/width of that across."""
    x = 0.5 * (1 + lobatto(n))
    N = n ** D
    height *= rng.uniform(0.7, 1.4)
    z = x[np.arange(N) // n ** (D - 1)] * height
    size = np.array([width * height] * (D - 1) + [height])
    ja = np.zeros((N, D, D))
    ja[:, range(D), range(D)] = np.prod(size) / 2 ** (D - 1) / size
    ja[:, D - 1, 0] = -tilt * ja[:, D - 1, D - 1] * rng.uniform(0.5, 1, N)
    T = rng.uniform(220, 300) * (1 + 1e-3 * rng.uniform(-1, 1, N))
    fall = G * height / (287 * T.mean()) if octaves is None else octaves * np.log(2)
    p = 1e5 * np.exp(-fall * z / height) * np.exp2(scatter * rng.uniform(-1, 1, N))
    rho = p / (287 * T) * np.exp2(scatter * rng.uniform(-1, 1, N))
    v = wind * rng.uniform(-1, 1, (N, D))
    v[:, D - 1] /= width
    u = np.stack([rho, *(rho * v.T), p / (CP / CV - 1) + 0.5 * rho * (v * v).sum(1), G * z], 1)
    return u, ja, end_fluxes(D, n, u, ja)


def lobatto(n):
    r = np.polynomial.legendre.Legendre.basis(n - 1).deriv().roots().real
    return np.concatenate([[-1.0], np.sort(r), [1.0]])


def end_fluxes(D, n, u, ja, more=0.0):
    """Fluxes through the end faces at the nodes' states, their normal velocities changed by `more`."""
    out = []
    v = u[:, 1:1 + D] / u[:, :1]
    p = (CP / CV - 1) * (u[:, 1 + D] - 0.5 * (u[:, 1:1 + D] * v).sum(1))
    for f in range(2 * D):
        i = end_nodes(D, n, f)
        nrm = ja[i, f // 2] * (1 if f & 1 else -1)
        vn = (v[i] * nrm).sum(1) + more * np.linalg.norm(nrm, axis=1)
        F = u[i, :D + 2] * vn[:, None]
        F[:, 1:1 + D] += p[i, None] * nrm
        F[:, 1 + D] += p[i] * vn
        out.append(F)
    return np.concatenate(out)


@pytest.mark.parametrize("D,n", [(2, 2), (2, 3), (2, 4), (2, 6), (2, 8), (3, 3), (3, 4)])
@pytest.mark.parametrize("width", [1, 16, 300, 2000, 20000])
@pytest.mark.parametrize("wind,tilt", [(20.0, 0.0), (0.0, 0.0), (20.0, 0.01)])
def test_words_are_no_less_precise_than_fp64(host, D, n, width, wind, tilt):
    words, fp64 = [], []
    for seed in range(40 if D == 2 else 10):
        u, ja, sf = flat_element(D, n, width, wind, np.random.default_rng(seed), tilt)
        ok, ew, ef, _ = host(D, n, u, ja, sf)
        assert ok
        words.append((ew ** 2).mean(0))
        fp64.append((ef ** 2).mean(0))
    words, fp64 = np.sqrt(np.mean(words, 0)), np.sqrt(np.mean(fp64, 0))
    some = fp64 > 0  # at rest the fluxes of mass and energy vanish
    assert np.all(words[some] <= 1.25 * fp64[some]), words / fp64
    assert np.all(words[~some] == 0)


@pytest.mark.parametrize("D,n", [(2, 3), (2, 4), (2, 6), (3, 4)])
@pytest.mark.parametrize("octaves", [1, 2, 3, 4, 6, 8, 12, 16])
def test_thin_nodes_of_tall_elements(host, D, n, octaves):
    """Isothermal elements whose density falls by 2^octaves: up to 3 are taken in words, from 4 on in
    FP64, and no row of nodes loses more than a binary place to the FP64 form."""
    words, fp64 = [], []
    for seed in range(40 if D == 2 else 6):
        u, ja, sf = flat_element(D, n, 20, 20.0, np.random.default_rng(seed), octaves=octaves)
        ok, ew, ef, _ = host(D, n, u, ja, sf)
        assert ok if octaves <= 3 else not ok
        if not ok:
            return
        words.append((ew ** 2).reshape(n, -1, D + 2).mean(1))
        fp64.append((ef ** 2).reshape(n, -1, D + 2).mean(1))
    assert np.all(np.mean(words, 0) <= 4 * np.mean(fp64, 0))


@pytest.mark.parametrize("n", range(2, 9))
def test_end_fluxes_have_their_exact_weight(host, n):
    """An element at rest takes its mass fluxes through the faces over the end weight 2 / (n (n - 1)):
    one rounding, and 2^-60 of the largest for the words (four places of scale)."""
    rng = np.random.default_rng(n)
    u, ja, sf = flat_element(2, n, 4, 0.0, rng)
    sf[:] = 0
    sf[:, 0] = rng.uniform(0.5, 1, len(sf))
    ok, ew, _, _ = host(2, n, u, ja, sf)
    limit = 0.5 * np.spacing(sf.reshape(4, n, 4)[..., 0] * (n * (n - 1) / 2)) + n * n * 2.0 ** -60
    assert ok
    for f in range(4):
        inner = end_nodes(2, n, f)[1:-1]  # the corners have a second face
        assert np.all(np.abs(ew[inner, 0]) <= limit[f, 1:-1])


@pytest.mark.parametrize("D,n", [(2, 2), (2, 5), (2, 8), (3, 3)])
def test_words_do_not_overflow(host, D, n):
    rng = np.random.default_rng(10 * D + n)
    for _ in range(60):
        u, ja, sf = flat_element(D, n, 2.0 ** rng.uniform(-3, 16), 10.0 ** rng.uniform(-6, 3), rng,
                                 tilt=rng.choice([0.0, 0.3]), scatter=rng.choice([0.0, 1.0]),
                                 height=10.0 ** rng.uniform(1, 4.5))
        turn = np.linalg.qr(rng.normal(size=(D, D)))[0]
        ja = np.ascontiguousarray(ja @ turn.T) * 2.0 ** rng.integers(-40, 20)
        u[:, 1:1 + D] = u[:, 1:1 + D] @ turn.T
        u[:, :2 + D] *= 2.0 ** rng.integers(-40, 40)
        sf = end_fluxes(D, n, u, ja, rng.choice([0.0, 10.0 ** rng.uniform(-6, 3)]))
        ok, ew, _, size = host(D, n, np.ascontiguousarray(u), ja, np.ascontiguousarray(sf))
        assert not ok or np.all(np.abs(ew).max(0) <= 1e-9 * size.max(0))


def face_pressure(n, u, ja, f):
    i = end_nodes(2, n, f)
    return (GAMMA - 1) * u[i, 3, None] * ja[i, f // 2] * (1 if f & 1 else -1)


@pytest.mark.gpu
@pytest.mark.parametrize("polydeg", [1, 2, 3, 5, 7])
@pytest.mark.parametrize("width", [1, 300, 20000])
def test_rest_on_flat_meshes(tg, gpu_lib, polydeg, width):
    n, nx, ny, lz = polydeg + 1, 3, 4, 10000.0
    lx = width * lz / ny * nx
    eq = tg.CompressibleEulerEnergyEquationsWithGravity2D(c_p=CP, c_v=CV, gravity=G)
    solver = tg.DGSEM(polydeg, (tg.FluxLMARS(340.0), tg.flux_zero), tg.VolumeIntegralFluxDifferencing(
        (tg.flux_ranocha, tg.flux_nonconservative_waruszewski_etal)))
    wall = tg.boundary_condition_slip_wall
    semi = tg.SemidiscretizationHyperbolic(
        tg.StructuredMesh((nx, ny), (0.0, 0.0), (lx, lz), periodicity=(True, False)), eq, None, solver,
        boundary_conditions={"y_neg": wall, "y_pos": wall})
    x = np.asarray(semi.node_coordinates)  # [element, j, i, 2]
    # the same values on both sides of every face: at rest the interface flux is the pressure alone
    p = 1e5 * np.exp(-G * x[..., 1] / (287 * 250.0)) * (1 + 1e-3 * np.cos(2 * np.pi * np.round(
        x[..., 0] / lx, 9)))
    u = np.zeros(x.shape[:-1] + (5,))
    u[..., 0], u[..., 3], u[..., 4] = p / (287 * 250.0), p / (CP / CV - 1), G * x[..., 1]
    u = np.ascontiguousarray(u)
    du = semi.rhs(u)
    assert semi.status() == 0
    # the discretisation's own operator, weights and metric terms, as the kernels get them
    S, w0 = semi.solver.basis.derivative_split, L(semi.solver.basis.weights[0])
    S = np.where(np.eye(n, dtype=bool), 0, S).astype(L)
    ja = np.asarray(semi.contravariant_vectors).reshape(-1, n * n, 2, 2).astype(L)
    ij = np.asarray(semi.inverse_jacobian).reshape(-1, n * n).astype(L)
    flat = u.reshape(-1, n * n, 5).astype(L)
    sf = np.zeros((nx * ny, 4, n, 4), L)
    if_e, if_f, _, bd_e, bd_f = (np.asarray(a, np.int64) for a in semi._H.connectivity_arrays[:5])
    for (e, e1), (f, f1) in zip(if_e, if_f):  # outward pressure fluxes, normals of the first side
        F = face_pressure(n, flat[e], ja[e], f)
        sf[e, f, :, 1:3], sf[e1, f1, :, 1:3] = F, -F
    for e, f in zip(bd_e, bd_f):
        sf[e, f, :, 1:3] = face_pressure(n, flat[e], ja[e], f)
    want = np.stack([-exact(2, n, flat[e], ja[e], sf[e], (S, w0))[0][:, 1] * ij[e]
                     for e in range(nx * ny)])
    size = np.abs(ja[..., 0, 0] * ij).max()
    bound = (n + 2) * 2.0 ** -53 * (np.abs(S).sum(1).max() + 1 / w0) * p.max() * size
    error = np.abs(du[..., 1].reshape(want.shape) - want)
    assert error.max() <= bound, float(error.max() / bound)
    semi.close()
