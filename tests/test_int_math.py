"""The integer-pipe functions of csrc/int_math.cuh (reciprocal, quotient, roots, logarithm,
exponential, power and the factors of the logarithmic means) against extended precision.

On the CPU the header is compiled with the host compiler: the same word arithmetic as on the
device but for the 24-bit seeds of the reciprocal and reciprocal square root.  The seeds' own error
(one and two last places) is inside the margin by which the code lowers them, so the bounds hold on
the device too, where `tag_eval_means` kinds 7 and 8 check them.  Bounds, in units of the result's
last place: one rounding (0.5) plus the fixed-point error (2^-58 relative: 0.03) for the algebraic
functions; 0.25 for exp, whose argument keeps 54 fraction bits from 16 up and 60 below; the mean factors 0.5 plus
the error of two node logarithms (2^-53 each, times |factor'| < 0.36)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "trixiatmo.jl_gb300", "csrc")
HARNESS = r"""
#include "int_math.cuh"
using namespace tag;
extern "C" void evaluate(int f, long n, const double* x, const double* y, double* out) {
  for (long i = 0; i < n; ++i) {
    const u64 yq = (u64)(y[i] * 2305843009213693952.0);
    switch (f) {
      case 0: out[i] = int_rcp(x[i]); break;
      case 1: out[i] = int_div(x[i], y[i]); break;
      case 2: out[i] = int_sqrt(x[i]); break;
      case 3: out[i] = int_rsqrt(x[i]); break;
      case 4: out[i] = (double)log2_fixed(x[i]) / 4503599627370496.0; break;
      case 5: out[i] = int_pow(x[i], y[i], yq); break;
      case 6: out[i] = int_exp(x[i]); break;
      case 7: case 8: {
        const u64 a = magnitude(log2_fixed(y[i]) - log2_fixed(x[i]));
        out[i] = !series_in_range(a) ? -1.0
                 : f == 7 ? ln_mean_factor(log_square(a)) : inv_ln_mean_factor(log_square(a));
        break;
      }
      case 9: out[i] = int_log2_ratio(x[i], (i64)(y[i] * 288230376151711744.0)); break;
    }
  }
}
"""
L = np.longdouble


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("int_math")
    src, lib = d / "harness.cpp", d / "harness.so"
    src.write_text(HARNESS)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(cuda, "include"),
                    "-I", CSRC, str(src), "-o", str(lib)], check=True)
    fn = ctypes.CDLL(str(lib)).evaluate
    dp = np.ctypeslib.ndpointer(np.float64, flags="C")
    fn.argtypes = [ctypes.c_int, ctypes.c_long, dp, dp, dp]

    def call(f, x, y=None):
        x = np.ascontiguousarray(x, dtype=np.float64)
        y = np.ones_like(x) if y is None else np.ascontiguousarray(y, dtype=np.float64)
        out = np.empty_like(x)
        fn(f, x.size, x, y, out)
        return out
    return call


def sample(seed=3, n=200_000):
    """Positive normal values: all magnitudes, and both ends of the binades where the seeds and the
    packing change (1 + k ulp, 2 - k ulp)."""
    rng = np.random.default_rng(seed)
    m = rng.uniform(1, 2, n)
    m[: n // 4] = 1 + rng.integers(0, 64, n // 4) * 2.0 ** -52
    m[n // 4: n // 2] = 2 - rng.integers(1, 65, n // 4) * 2.0 ** -52
    return m * 2.0 ** rng.integers(-300, 300, n)


def ulps(got, want):
    return np.max(np.abs(got.astype(L) - want) / np.spacing(np.abs(want.astype(np.float64))))


def test_algebraic_functions(host):
    x, y = sample(), sample(4)
    assert ulps(host(0, x), 1 / x.astype(L)) <= 0.53
    assert ulps(host(0, -x), -1 / x.astype(L)) <= 0.53
    assert ulps(host(1, x, y), x.astype(L) / y.astype(L)) <= 0.53
    assert ulps(host(2, x), np.sqrt(x.astype(L))) <= 0.53
    assert ulps(host(3, x), 1 / np.sqrt(x.astype(L))) <= 0.53


def test_exponential_and_logarithm(host):
    x = sample()
    assert np.max(np.abs(host(4, x).astype(L) - np.log2(x.astype(L)))) <= 2.0 ** -52.9 + 300 * 2.0 ** -53
    near = x * 2.0 ** -np.floor(np.log2(x))
    assert np.max(np.abs(host(4, near).astype(L) - np.log2(near.astype(L)))) <= 1.1 * 2.0 ** -53
    rng = np.random.default_rng(5)
    g = rng.uniform(1.0, 2.5, x.size)
    s = x ** 0.1  # keeps the powers normal
    q = np.floor(g * 2.0 ** 61) / L(2) ** 61
    assert ulps(host(5, s, g), s.astype(L) ** q) <= 0.7
    e = rng.uniform(-500, 500, x.size) * 10.0 ** rng.uniform(-8, 0, x.size)
    assert ulps(host(6, e), np.exp(e.astype(L))) <= 0.7
    r = 273.15 * rng.uniform(0.3, 3, x.size)
    ref = np.floor(np.log2(273.15) * 2.0 ** 58) / 2.0 ** 58
    want = np.log2(r.astype(L)) - L(ref)
    off = np.abs(host(9, r, np.full_like(r, ref)).astype(L) - want)
    assert np.all(off <= 2.0 ** -57 + 0.5 * np.spacing(np.abs(want.astype(np.float64))))


def test_mean_factors(host):
    rng = np.random.default_rng(6)
    x = sample()
    ratio = np.exp2(rng.uniform(-1, 1, x.size) * 10.0 ** rng.uniform(-9, 0, x.size))
    y = x * ratio
    d = np.log(y.astype(L) / x.astype(L))
    with np.errstate(invalid="ignore"):
        ln = np.where(d == 0, L(1), np.tanh(d / 2) / (d / 2))
        inv = np.where(d == 0, L(1), d / np.sinh(d))
    for f, want in ((7, ln), (8, inv)):
        got = host(f, x, y)
        on = got >= 0
        assert on.mean() > 0.99
        assert np.max(np.abs(got[on].astype(L) - want[on])) <= 1.3 * 2.0 ** -53
    assert np.all(host(7, x, x) == 1) and np.all(host(8, x, x) == 1)
    assert np.all(host(7, x, 2.1 * x) == -1)


def test_special_values(host):
    """Zeros, infinities, NaN, negative and subnormal arguments come out as the CUDA functions'."""
    x = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, -1.0, 5e-324, 1e-310, 1e308, -1e-308])
    with np.errstate(all="ignore"):
        for f, want in ((0, 1 / x), (2, np.sqrt(x)), (3, 1 / np.sqrt(x)), (1, x / 3.0), (6, np.exp(x))):
            got = host(f, x, np.full_like(x, 3.0))
            same = (got == want) | (np.isnan(got) & np.isnan(want)) | (np.abs(got - want) <= np.spacing(np.abs(want)))
            assert np.all(same), (f, got, want)
    assert np.allclose(host(4, np.array([5e-324, 1e-310])), [-1074, np.log2(1e-310)], atol=1e-12)


@pytest.mark.gpu
def test_device_functions(tg, gpu_lib):
    from test_gpu_means import device
    x, y = sample(), sample(9)
    gamma = (1004.0, 717.0)
    rcp, rsq = device(tg, 7, x, y, gamma)
    assert ulps(rcp, 1 / x.astype(L)) <= 0.53 and ulps(rsq, 1 / np.sqrt(y.astype(L))) <= 0.53
    s = x ** 0.1
    e = np.random.default_rng(7).uniform(-500, 500, x.size)
    g = L(np.floor(np.float64(1004.0 / 717.0) * 2.0 ** 61)) / L(2) ** 61
    pw, ex = device(tg, 8, s, e, gamma)
    assert ulps(pw, s.astype(L) ** g) <= 0.7 and ulps(ex, np.exp(e.astype(L))) <= 0.7
