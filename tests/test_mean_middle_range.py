"""The means' factors of values more than a factor of two apart (csrc/int_math.cuh, middle range:
up to a factor of 256): on the CPU against extended precision at given logarithms' differences, to
one rounding of the double and 2^-57 of the words; on the GPU the potential-temperature right-hand
side, whose Stolarsky and logarithmic means take them, against the CPU oracle for neighbours on both
sides of the range's ends."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from test_int_math import CSRC

HARNESS = r"""
#include "int_math.cuh"
using namespace tag;
extern "C" void middle(int f, long n, const i64* d, double gamma, double* out) {
  const u64 g = pow_exponent(gamma), s = (u64)ldexpl(2.0L * ((long double)gamma - 1.0L) / gamma, 64);
  for (long i = 0; i < n; ++i) {
    const u64 a = magnitude(d[i]);
    out[i] = !middle_range(a) ? -1.0
             : middle_factor(f == 0 ? ln_mean_deficit_middle(a)
                             : f == 1 ? inv_ln_mean_deficit_middle(a)
                                      : stolarsky_deficit_middle(a, g, s));
  }
}
"""
L = np.longdouble


@pytest.fixture(scope="module")
def middle(tmp_path_factory):
    d = tmp_path_factory.mktemp("middle")
    src, lib = d / "harness.cpp", d / "harness.so"
    src.write_text(HARNESS)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(cuda, "include"),
                    "-I", CSRC, str(src), "-o", str(lib)], check=True)
    fn = ctypes.CDLL(str(lib)).middle
    fn.argtypes = [ctypes.c_int, ctypes.c_long, np.ctypeslib.ndpointer(np.int64, flags="C"),
                   ctypes.c_double, np.ctypeslib.ndpointer(np.float64, flags="C")]

    def call(f, d, gamma=1.4):
        out = np.empty(d.size)
        fn(f, d.size, d, gamma, out)
        return out
    return call


def differences():
    """log2_fixed differences (Q11.52) in [1, 8): spread, at the ends and around the integers."""
    rng = np.random.default_rng(1)
    d = rng.integers(1 << 52, 8 << 52, 100_000)
    whole = np.arange(1, 8) * (1 << 52)
    near = (whole[:, None] + rng.integers(-1000, 1000, (7, 50))).ravel()
    d = np.concatenate([d, whole, near, [(8 << 52) - 1]])
    d = d[d >= 1 << 52]
    return np.concatenate([d, -d]).astype(np.int64)


@pytest.mark.parametrize("gamma", [1004 / 717, 5 / 3, 1.3, 1.9])
def test_factors(middle, gamma):
    d = differences()
    D = np.abs(d).astype(L) / L(2) ** 52
    x = D * np.log(L(2)) / 2
    g = L(gamma)
    wants = (np.tanh(x) / x, 2 * x / np.sinh(2 * x),
             (g - 1) / g * np.sinh(g * x) / (np.sinh((g - 1) * x) * np.cosh(x)))
    for f, want in enumerate(wants):
        got = middle(f, d, gamma)
        # half a last place of the double, and the words' error
        limit = 0.5 * np.spacing(want.astype(np.float64)) + 2.0 ** -56 * want
        assert np.all(np.abs(got.astype(L) - want) <= limit), f
    assert np.all(middle(0, np.array([8 << 52, -(8 << 52), 1 << 62], np.int64)) == -1)


@pytest.mark.gpu
@pytest.mark.parametrize("volume,nc", [("tec", "souza"), ("ec", "waruszewski"), ("tec", "artiano"),
                                       ("etec", "waruszewski")])
@pytest.mark.parametrize("octaves", [1.05, 4.0, 8.5])
def test_potential_temperature_rhs(tg, orc, gpu_lib, volume, nc, octaves):
    """Neighbouring values up to 2^octaves apart, each variable within 1e-11 of its max norm (the
    parity tests' tolerance)."""
    from test_gpu_pt import C_LMARS, make_pt
    eq, mesh, semi = make_pt(tg, polydeg=3, volume=volume, nc=nc)
    u = semi.compute_coefficients()
    rng = np.random.default_rng(int(octaves * 100))
    for v in (0, 3):
        f = np.exp2(rng.uniform(-octaves / 2, octaves / 2, u.shape[:-1]))
        u[..., v] *= f
        if v == 0:
            u[..., 1] *= f
            u[..., 2] = u[..., 0] * rng.uniform(-5, 5, f.shape)
    du = semi.rhs(u)
    ref = orc.PotTemp2D(3, 8, 6, 0.0, 300000.0, 0.0, 10000.0, True, False,
                        volume={"tec": 0, "ec": 1, "etec": 2}[volume],
                        nc={"waruszewski": 0, "artiano": 1, "souza": 2}[nc], wall_kind=1,
                        c_lmars=C_LMARS).rhs(u)
    for v in range(4):
        assert np.abs(du[..., v] - ref[..., v]).max() <= 1e-11 * np.abs(ref[..., v]).max(), v
    assert semi.status() == 0
    semi.close()
