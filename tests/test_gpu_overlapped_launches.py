"""Runs whose stage kernels overlap (meshes up to 24,576 nodes) and runs just above, against the same
steps driven from the host, where every right-hand side is waited for: a kernel that read what its
predecessor had not yet written would be off by a whole stage.

Tolerance: both sides evaluate the same right-hand sides; the stage update rounds three times per
stage on the host and once or twice on the device.  A pressure that differs by 1e-16 of itself
changes the momentum by 1e-16 c/v of its own size; with v above c/1000 and 60 stages that is 6e-12,
so 1e-11 of each variable's largest value.  (A stage too few or too many is off by 1e-4 and more.)
"""
import numpy as np
import pytest

from test_gpu_cov_swe import make_semi as make_swe
from test_gpu_euler2d import make_semi as make2d
from test_gpu_euler3d import make_semi as make3d
from test_oracle_golden_3d import perturb3d

pytestmark = pytest.mark.gpu


def build(tg, kind, size):
    if kind == "2d":
        eq, semi = make2d(tg, *size, 3)
        return semi, tg.seeded_perturbation(semi.compute_coefficients(), eq, seed=1)
    if kind == "3d":
        eq, _, semi = make3d(tg, *size, 3)
        return semi, perturb3d(semi.compute_coefficients(), eq, seed=1)
    semi = make_swe(tg, "rossby_haurwitz", k=size, polydeg=3)[2]
    return semi, np.asarray(semi.compute_coefficients()).reshape(semi.shape)


@pytest.mark.parametrize("kind,size", [("2d", (3, 2)), ("2d", (48, 32)), ("2d", (49, 32)),
                                       ("3d", (3, 3)), ("3d", (4, 5)), ("swe", 5), ("swe", 16),
                                       ("swe", 17)])
def test_runs_match_host_driven_steps(tg, gpu_lib, kind, size):
    semi, u0 = build(tg, kind, size)
    semi.set_state(u0)
    dt = 0.3 * float(np.min(semi.max_dt()))
    steps = 20
    semi.rk_steps(steps, fixed_dt=dt, method="SSPRK33")
    got = np.asarray(semi.get_state()).reshape(u0.shape)
    u = u0.copy()
    for _ in range(steps):
        w = u + dt * semi.rhs(u).reshape(u0.shape)
        w = 0.75 * u + 0.25 * (w + dt * semi.rhs(w).reshape(u0.shape))
        u = u / 3.0 + 2.0 / 3.0 * (w + dt * semi.rhs(w).reshape(u0.shape))
    for v in range(u0.shape[-1]):
        assert np.abs(got[..., v] - u[..., v]).max() <= 1e-11 * np.abs(u[..., v]).max(), v
    semi.close()
