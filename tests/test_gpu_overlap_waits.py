"""Right-hand sides of two unrelated states, back to back on small meshes (whose interface and element
kernels overlap): an element kernel that did not wait for its own interface kernel would take the
other state's surface fluxes, an interface kernel that did not wait would change them under the
element kernel before.  Both states' results are the CPU oracle's, at the parity tests' tolerance (the
other state's surface fluxes would be off by a tenth and more), and the same bits in every repetition."""
import numpy as np
import pytest

from test_gpu_cov_swe import make_semi as make_swe
from test_gpu_cov_swe import oracle_for
from test_gpu_cov_swe import perturbed as perturb_swe
from test_gpu_euler2d import make_semi as make2d
from test_gpu_euler2d import oracle_case
from test_gpu_euler3d import make_semi as make3d
from test_gpu_euler3d import solver_basis
from test_gpu_moist import bubble_semi, moist_state
from test_gpu_pt import C_LMARS, make_pt
from test_gpu_pt import perturbed as perturb_pt
from test_gpu_rainy import make_rainy, moving, solved_state
from test_oracle_golden_3d import oracle_3d, perturb3d

pytestmark = pytest.mark.gpu


def case(tg, orc, kind):
    if kind == "2d":
        eq, semi = make2d(tg, 16, 8, 3)
        make = lambda s: tg.seeded_perturbation(semi.compute_coefficients(), eq, seed=s)  # noqa: E731
        return semi, make, oracle_case(orc, 16, 8, 3).rhs
    if kind == "3d":
        eq, mesh, semi = make3d(tg, 2, 2, 3)
        make = lambda s: perturb3d(semi.compute_coefficients(), eq, seed=s)  # noqa: E731
        return semi, make, oracle_3d(orc, tg, 3, semi.contravariant_vectors, semi.inverse_jacobian,
                                     semi.node_coordinates, mesh.connectivity(solver_basis(semi))).rhs
    if kind == "pt":
        semi = make_pt(tg, polydeg=3)[2]
        return semi, lambda s: perturb_pt(semi.compute_coefficients(), s), orc.PotTemp2D(
            3, 8, 6, 0.0, 300000.0, 0.0, 10000.0, True, False, volume=0, nc=0, wall_kind=1,
            c_lmars=C_LMARS).rhs
    if kind == "moist":
        eq, _, semi = bubble_semi(tg, 3)
        return semi, lambda s: moist_state(eq, semi.compute_coefficients(), seed=s), orc.Moist2D(
            3, 8, 6, 0.0, 20000.0, -5000.0, 15000.0, True, False, surface_kind=0, source_kind=1,
            wall_kind=1).rhs
    if kind == "rainy":
        semi = make_rainy(tg, 8, 4, 3)[1]
        make = lambda s: solved_state(orc, moving(semi.compute_coefficients(), seed=s))  # noqa: E731
        return semi, make, orc.Rainy2D(3, 8, 4, 0.0, 20000.0, 0.0, 10000.0, True, False).rhs
    eq, mesh, semi, fluxes, _ = make_swe(tg, kind, k=4, polydeg=3)
    make = lambda s: perturb_swe(np.asarray(semi.compute_coefficients()), s)  # noqa: E731
    return semi, make, oracle_for(orc, semi, mesh, eq, fluxes).rhs


@pytest.mark.parametrize("kind", ["2d", "3d", "pt", "moist", "rainy", "rossby_haurwitz",
                                  "isolated_mountain"])
def test_alternating_states(tg, orc, gpu_lib, kind):
    torch = pytest.importorskip("torch")
    semi, make, reference = case(tg, orc, kind)
    states = [np.ascontiguousarray(make(s), dtype=np.float64) for s in (1, 2)]
    states[1].reshape(-1, states[1].shape[-1])[:] *= 1.1  # all variables; geopotential and T below
    if kind in ("2d", "3d", "pt"):
        states[1][..., -1] = states[0][..., -1]
    if kind == "rainy":
        states[1][..., 6:] = states[0][..., 6:]
        states[1] = solved_state(orc, states[1])
    u = [torch.from_numpy(s).cuda() for s in states]
    du = [[torch.zeros_like(v) for v in u] for _ in range(12)]
    semi.rhs_device(u[0].data_ptr(), du[0][0].data_ptr())  # (chooses the tile)
    torch.cuda.synchronize()
    for d in du:  # nothing waits between the calls
        for k in (0, 1):
            semi.rhs_device(u[k].data_ptr(), d[k].data_ptr())
    torch.cuda.synchronize()
    semi.rhs(states[0])  # the handle's own stream is done, too
    tol = 1e-10 if kind == "rainy" else 1e-11
    for k in (0, 1):
        want = np.asarray(reference(states[k])).reshape(-1, states[k].shape[-1])
        got = du[-1][k].cpu().numpy().reshape(want.shape)
        for v in range(want.shape[1]):
            assert np.abs(got[:, v] - want[:, v]).max() <= tol * np.abs(want[:, v]).max(), (k, v)
        for d in du:
            assert torch.equal(d[k], du[-1][k])
    semi.close()
