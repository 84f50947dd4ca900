"""The element kernels' tiles: every one that the autotuner tries can be set, gives the same bits, and
the one it keeps can be read back; the reported CTA width is the one that is launched (no more threads
than the kernel's registers allow)."""
import numpy as np
import pytest

from test_gpu_cov_swe import make_semi as make_swe
from test_gpu_euler2d import make_semi as make2d
from test_gpu_euler3d import make_semi as make3d
from test_gpu_pt3d import make_pt3d
from test_gpu_rainy import make_rainy
from test_oracle_golden_3d import perturb3d

pytestmark = pytest.mark.gpu


def case(tg, kind, polydeg):
    if kind == "2d":
        eq, semi = make2d(tg, 6, 5, polydeg)
        return semi, tg.seeded_perturbation(semi.compute_coefficients(), eq, seed=polydeg)
    if kind == "rainy":
        semi = make_rainy(tg, 6, 5, polydeg)[1]
        return semi, semi.compute_coefficients()
    if kind == "3d":
        eq, _, semi = make3d(tg, 2, 2, polydeg)
    else:
        semi = make_pt3d(tg, 2, 2, polydeg)[2]
        return semi, semi.compute_coefficients()
    return semi, perturb3d(semi.compute_coefficients(), eq, seed=polydeg)


@pytest.mark.parametrize("kind,polydeg", [("2d", 1), ("2d", 3), ("2d", 7), ("rainy", 3), ("3d", 2),
                                          ("3d", 3), ("3d", 5), ("pt3d", 3)])
def test_same_bits_for_every_tile(tg, gpu_lib, kind, polydeg):
    semi, u = case(tg, kind, polydeg)
    assert semi.tile()[0] == 0
    want = semi.rhs(u)  # the autotuner's choice
    epb, items = semi.tile()
    width = semi.cta_threads()
    semi.set_tile(epb, items)
    assert semi.tile() == (epb, items) and semi.cta_threads() == width
    tried = 0
    for epb in (1, 2, 3, 4, 6, 8, 12, 16):
        for items in range(1, 7 if kind.endswith("3d") else 4):
            try:
                semi.set_tile(epb, items)
            except RuntimeError:  # too large for one CTA
                continue
            assert semi.cta_threads() % 32 == 0
            assert np.array_equal(semi.rhs(u), want), (epb, items)
            tried += 1
    assert tried >= 6
    with pytest.raises(RuntimeError):
        semi.set_tile(1, 7 if kind.endswith("3d") else 4)
    semi.close()


def test_reported_width_is_launched(tg, gpu_lib):
    """Ten elements of degree 3 are 960 work items; the element kernel of the 3D energy equations holds
    more than 72 registers per thread, so no more than 65536 / 72 threads fit."""
    semi, u = case(tg, "3d", 3)
    semi.set_tile(10, 1)
    assert semi.cta_threads() <= 65536 // 72
    semi.rhs(u)
    semi.close()


@pytest.mark.parametrize("trees,threads", [(5, 128), (64, 256)])
def test_covariant_width(tg, gpu_lib, trees, threads):
    semi = make_swe(tg, "rossby_haurwitz", k=trees, polydeg=3)[2]
    assert semi.cta_threads() == threads
    semi.close()
