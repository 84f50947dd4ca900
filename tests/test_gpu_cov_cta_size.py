"""The covariant element kernel's CTA size is chosen by the mesh (128 or 256 threads per CTA): a member
alone (few CTAs: 128) and the same member inside an ensemble large enough for 256 evaluate the same
right-hand side, bit for bit, at element sizes that fill the CTAs and that do not."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("polydeg", [1, 3, 5, 6, 7])
def test_same_bits_for_both_sizes(tg, gpu_lib, polydeg):
    cv = tg.covariant
    eq = cv.CovariantShallowWaterEquations2D(9.80616, 7.292e-5)
    ic = cv.transform_initial_condition(cv.initial_condition_rossby_haurwitz, eq)
    solver = tg.DGSEM(polydeg, tg.flux_lax_friedrichs, tg.VolumeIntegralWeakForm())
    small = cv.P4estMeshCubedSphere2D(5, 6.37122e6, polydeg=polydeg)
    big = cv.P4estMeshCubedSphere2D(40, 6.37122e6, polydeg=7)
    src = cv.source_terms_geometric_coriolis
    alone = tg.SemidiscretizationHyperbolic(small, eq, ic, solver, source_terms=src)
    u = np.ascontiguousarray(alone.compute_coefficients(), dtype=np.float64).reshape(-1)
    want = np.asarray(alone.rhs(u.reshape(alone.shape))).reshape(-1)
    both = tg.SemidiscretizationCovariantEnsemble(
        [small, big], eq, [ic, ic],
        [solver, tg.DGSEM(7, tg.flux_lax_friedrichs, tg.VolumeIntegralWeakForm())], source_terms=src)
    w = np.ascontiguousarray(both.compute_coefficients(), dtype=np.float64).reshape(-1)
    w[: u.size] = u
    got = np.asarray(both.rhs(w.reshape(both.shape))).reshape(-1)[: u.size]
    assert np.array_equal(got, want)
    alone.close()
    both.close()
