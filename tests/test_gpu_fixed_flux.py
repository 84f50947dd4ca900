"""The element kernels' fixed-point volume integral (csrc/fixed_flux.cuh) where its words could go
wrong: node values beyond a factor of two (the means' far branch), states at rest, one moving node in
an element at rest, magnitudes near and beyond the scales' range (2^+-150: the FP64 form), and bad
states, which take the FP64 form and set the status word.

Against the CPU oracle at the parity tests' tolerance: every variable within 1e-11 of its own max
norm."""
import numpy as np
import pytest

from test_gpu_euler2d import make_semi as make2d
from test_gpu_euler2d import oracle_case
from test_gpu_euler3d import make_semi as make3d
from test_gpu_euler3d import solver_basis
from test_oracle_golden_3d import oracle_3d, perturb3d

pytestmark = pytest.mark.gpu


def case(tg, orc, dim, polydeg):
    if dim == 2:
        eq, semi = make2d(tg, 6, 5, polydeg)
        u = tg.seeded_perturbation(semi.compute_coefficients(), eq, seed=polydeg)
        return eq, semi, u, oracle_case(orc, 6, 5, polydeg).rhs
    eq, mesh, semi = make3d(tg, 2, 2, polydeg)
    u = perturb3d(semi.compute_coefficients(), eq, seed=polydeg)
    o = oracle_3d(orc, tg, polydeg, semi.contravariant_vectors, semi.inverse_jacobian,
                  semi.node_coordinates, mesh.connectivity(solver_basis(semi)))
    return eq, semi, u, o.rhs


def prims(eq, u):
    p = eq.cons2prim(u)
    return list(p) if isinstance(p, tuple) else [p[..., k] for k in range(p.shape[-1])]


def check(semi, u, ref, tol=1e-11):
    du = semi.rhs(u)
    want = ref(u)
    for v in range(u.shape[-1] - 1):
        s = np.abs(want[..., v]).max()
        assert np.abs(du[..., v] - want[..., v]).max() <= tol * s, v
    assert semi.status() == 0


@pytest.mark.parametrize("dim,polydeg", [(2, 1), (2, 3), (2, 4), (2, 7), (3, 2), (3, 5)])
@pytest.mark.parametrize("kind", ["factor", "rest", "one_node", "large", "beyond", "thin"])
def test_fixed_point_volume_integral(tg, orc, gpu_lib, dim, polydeg, kind):
    eq, semi, u, ref = case(tg, orc, dim, polydeg)
    q = prims(eq, u)
    rho, v, p, phi = q[0], q[1:-2], q[-2], q[-1]
    rng = np.random.default_rng(polydeg)
    if kind == "factor":  # neighbours up to a factor of 8 apart in density and pressure
        rho = rho * np.exp2(rng.uniform(-1.5, 1.5, rho.shape))
        p = p * np.exp2(rng.uniform(-1.5, 1.5, rho.shape))
    elif kind == "rest":
        v = [0 * w for w in v]
        rho = rho * (1 + 0.1 * rng.uniform(-1, 1, rho.shape))
    elif kind == "one_node":
        at = np.zeros(rho.shape, bool)
        at.reshape(rho.shape[0], -1)[:, 1] = True
        v = [np.where(at, w, 0.0) for w in v]
    elif kind == "large":  # inside the scales' range
        rho, p, phi = rho * 2.0 ** 60, p * 2.0 ** 80, phi * 2.0 ** 20
        v = [w * 2.0 ** 10 for w in v]
    elif kind == "beyond":  # outside it: the FP64 form
        rho, p = rho * 2.0 ** 160, p * 2.0 ** 160
    elif kind == "thin":
        rho, p = rho * 2.0 ** -120, p * 2.0 ** -120
    check(semi, np.ascontiguousarray(eq.prim2cons(rho, *v, p, phi)), ref)
    semi.close()


@pytest.mark.parametrize("dim", [2, 3])
def test_bad_states_set_the_status(tg, orc, gpu_lib, dim):
    eq, semi, u, _ = case(tg, orc, dim, 3)
    nv = u.shape[-1]
    for bad, bit in ((np.nan, tg._lib.TAG_S_NAN), (np.inf, tg._lib.TAG_S_NAN),
                     (-1.0, tg._lib.TAG_S_NEG_DENSITY)):
        w = u.copy()
        w.reshape(-1, nv)[nv * 7, 0] = bad
        semi.rhs(w)
        assert semi.status() & bit, bad
    w = u.copy()
    w.reshape(-1, nv)[11, nv - 2] = -1.0
    semi.rhs(w)
    assert semi.status() & tg._lib.TAG_S_NEG_PRESSURE
    semi.rhs(u)
    assert semi.status() == 0
    semi.close()
