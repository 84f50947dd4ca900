"""The reported CTA width of the element kernels is the one that is launched (no more threads than the
kernel's registers allow)."""
import pytest

from test_gpu_cov_swe import make_semi as make_swe
from test_gpu_euler3d import make_semi as make3d

pytestmark = pytest.mark.gpu


def test_reported_width_is_launched(tg, gpu_lib):
    """Ten elements of degree 3 are 960 work items; the element kernel of the 3D energy equations holds
    more than 72 registers per thread, so no more than 65536 / 72 threads fit."""
    semi = make3d(tg, 2, 2, 3)[2]
    u = semi.compute_coefficients()
    semi.set_tile(10, 1)
    assert semi.cta_threads() <= 65536 // 72
    semi.rhs(u)
    semi.close()


@pytest.mark.parametrize("trees,threads", [(5, 128), (64, 256)])
def test_covariant_width(tg, gpu_lib, trees, threads):
    semi = make_swe(tg, "rossby_haurwitz", k=trees, polydeg=3)[2]
    assert semi.cta_threads() == threads
    semi.close()
