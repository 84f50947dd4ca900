"""Logarithmic means of values that have none: negative and zero dry density, temperature and pressure.

The mean of two values of opposite sign is NaN (the logarithm of their ratio), so such a state has to
set TAG_S_NAN whatever the size of the values beside it; the mean of a value and zero is zero; the
mean of an inverse has no value at zero."""
import numpy as np
import pytest

from test_gpu_euler2d import make_semi as make2d
from test_gpu_euler3d import make_semi as make3d
from test_gpu_ie import make_ie
from test_gpu_moist import bubble_semi, moist_state
from test_gpu_pt import make_pt
from test_gpu_rainy import make_rainy
from test_int_math import host  # noqa: F401


def test_words_of_values_without_a_logarithm(host):  # noqa: F811
    x = np.array([1e-3, 0.05, 1.0, 1.1, 3.0, 1e200])
    for negative in (-x, -2.0 ** -1060 * x[:1]):
        assert np.allclose(host(4, negative), np.log2(-negative) + 1024, rtol=0, atol=1e-12)
    zero = host(4, np.zeros(1))[0]
    # beyond the series (one octave) and the middle range (eight) beside any other value
    assert np.all(np.abs(host(4, np.concatenate([x, -x, [5e-324]])) - zero) > 8)


def with_dry_density(eq, u, where, ratio):
    """Dry density `ratio` times the total one at `where`, at 290 K (no liquid)."""
    w = u.copy()
    rho = w[where][..., 0]
    v = w[where][..., 1:3] / rho[..., None]
    w[where + (4,)] = (1.0 - ratio) * rho
    w[where + (5,)] = 0.0
    qv = w[where + (4,)] / rho
    w[where + (3,)] = rho * (((1 - qv) * eq.c_vd + qv * eq.c_vv) * 290.0 + qv * eq.L_00 +
                             0.5 * (v ** 2).sum(-1))
    return w


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [0.05, 0.7, 1.0, 1.6, 2.5, 3.5, 40.0])
@pytest.mark.parametrize("ratio", [-0.05, -1e-3])
def test_negative_dry_density_sets_the_status(tg, gpu_lib, scale, ratio):
    eq, mesh, semi = bubble_semi(tg, 3)
    u = scale * moist_state(eq, semi.compute_coefficients(), seed=3)
    semi.rhs(u)
    assert semi.status() == 0
    w = with_dry_density(eq, u, (np.array([9]), np.array([1]), np.array([2])), ratio)
    du = semi.rhs(w)
    assert semi.status() & tg._lib.TAG_S_NAN
    assert not np.any(np.isfinite(du[9, 1, 2, :4]))
    semi.close()


@pytest.mark.gpu
def test_zero_dry_density(tg, orc, gpu_lib):
    eq, mesh, semi = bubble_semi(tg, 3)
    u = moist_state(eq, semi.compute_coefficients(), seed=3)
    w = with_dry_density(eq, u, (np.array([9]), np.array([1]), np.array([2])), 0.0)
    du = semi.rhs(w)
    assert semi.status() == 0
    ref = orc.Moist2D(3, 8, 6, 0.0, 20000.0, -5000.0, 15000.0, True, False, surface_kind=0,
                      source_kind=1, wall_kind=1).rhs(w)
    for v in range(6):
        assert np.abs(du[..., v] - ref[..., v]).max() <= 1e-11 * np.abs(ref[..., v]).max(), v
    # two on one line
    w = with_dry_density(eq, u, (np.array([9, 9]), np.array([1, 1]), np.array([2, 3])), 0.0)
    semi.rhs(w)
    assert semi.status() & tg._lib.TAG_S_NAN
    semi.close()


@pytest.mark.gpu
@pytest.mark.parametrize("kind,slot,value",
                         [("2d", 3, -1e5), ("2d", 3, 0.0), ("3d", 4, -1e5), ("3d", 4, 0.0),
                          ("ie", 3, -1e5), ("ie", 3, 0.0), ("moist", 3, -2e6),
                          ("tec", 3, -300.0), ("ec", 3, 0.0), ("etec", 3, 0.0),
                          ("tec", 3, 0.0), ("rainy", 8, -250.0), ("rainy", 8, 0.0)])
def test_temperature_and_pressure_without_a_mean(tg, gpu_lib, kind, slot, value):
    if kind == "2d":
        semi = make2d(tg, 6, 5, 3)[1]
    elif kind == "3d":
        semi = make3d(tg, 2, 2, 3)[2]
    elif kind == "ie":
        semi = make_ie(tg)[2]
    elif kind == "moist":
        semi = bubble_semi(tg, 3)[2]
    elif kind == "rainy":
        semi = make_rainy(tg, 8, 4, 3)[1]
    else:
        semi = make_pt(tg, polydeg=3, volume=kind)[2]
    u = semi.compute_coefficients()
    semi.rhs(u)
    assert semi.status() == 0
    flat = u.reshape(u.shape[0], -1, u.shape[-1])
    if kind == "rainy":  # not dry: the stored temperature is the node's
        flat[7, 6, 2] += 1e-6
    else:  # at rest, so that the pressure is the energy's alone
        flat[7, 6, 1:slot] = 0.0
    flat[7, 6, slot] = value
    semi.rhs(u)
    status = semi.status()
    assert status & tg._lib.TAG_S_NAN, status
    assert status & tg._lib.TAG_S_NEG_PRESSURE, status
    semi.close()
