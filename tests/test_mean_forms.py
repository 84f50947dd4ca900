"""The logarithmic means' factors in the forms that the kernels run, on the host against extended
precision, over every range and on both sides of each switch: the short series (values within 1.5 %),
the long one (a factor of two), the words' middle range (256) and beyond, and the fixed-point kernels'
choice among them (fx_ln_deficit, fx_inv_ln_deficit).

A factor 1 - c depends on the difference of two node logarithms (2^-53 each, and |factor'| < 0.36) and
on the words (2^-56); beyond 256 it is formed in FP64 from the values (four roundings)."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

from test_int_math import CSRC

HARNESS = r"""
#include "fixed_flux.cuh"
using namespace tag;
namespace tag { void set_last_error(const std::string&) {} }
extern "C" void factors(int f, long n, const double* x, const double* y, double* out) {
  for (long i = 0; i < n; ++i) {
    const i64 d = log2_fixed(y[i]) - log2_fixed(x[i]);
    const u64 a = magnitude(d);
    u64 c = 0;
    if (f < 2) {  // the kernels' choice, words of one scale
      const int e = std::ilogb(std::max(x[i], y[i])) + 1;
      const i64 wx = to_fixed(x[i], e), wy = to_fixed(y[i], e);
      c = f == 0 ? fx_ln_deficit(wx, wy, d) : fx_inv_ln_deficit(wx, wy, d);
    } else {
      const u64 z = log_square(a);
      if (!series_in_range(a) || (f < 4 && z >= kShortZ)) {
        out[i] = -1.0;
        continue;
      }
      c = f == 2 ? ln_mean_deficit_short(z) : f == 3 ? inv_ln_mean_deficit_short(z)
          : f == 4 ? ln_mean_deficit(z) : inv_ln_mean_deficit(z);
    }
    out[i] = 1.0 - std::ldexp((double)(c >> 1), -63);
  }
}
"""
L = np.longdouble


@pytest.fixture(scope="module")
def factors(tmp_path_factory):
    d = tmp_path_factory.mktemp("mean_forms")
    src, lib = d / "harness.cu", d / "harness.so"
    src.write_text(HARNESS)
    home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    nvcc = shutil.which("nvcc") or os.path.join(home, "bin", "nvcc")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-shared",
                    "-Xcompiler", "-fPIC", "-I", CSRC, str(src), "-o", str(lib)], check=True)
    fn = ctypes.CDLL(str(lib)).factors
    dp = np.ctypeslib.ndpointer(np.float64, flags="C")
    fn.argtypes = [ctypes.c_int, ctypes.c_long, dp, dp, dp]

    def call(f, x, y):
        out = np.empty_like(x)
        fn(f, x.size, x, y, out)
        return out
    return call


def pairs(low, high, n=20000):
    """Values whose logarithms to base 2 differ by [low, high], either one the larger."""
    rng = np.random.default_rng(int(1e4 * high))
    x = rng.uniform(0.5, 2.0, n)
    r = np.exp2(np.exp(rng.uniform(np.log(max(low, 1e-12)), np.log(high), n)))
    r[: n // 10] = np.exp2(high)
    y = x * np.where(rng.random(n) < 0.5, r, 1 / r)
    return x, y


SHORT = 2.0 ** -5.5  # kShortZ = 2^-11 of squared differences


@pytest.mark.parametrize("low,high", [(0, 1e-6), (1e-6, 0.5 * SHORT), (0.98 * SHORT, 1.02 * SHORT),
                                      (SHORT, 0.98), (0.98, 1.02), (1.0, 7.9), (7.9, 8.1), (8.1, 16)])
@pytest.mark.parametrize("inverse", [0, 1])
def test_factor_of_every_range(factors, low, high, inverse):
    x, y = pairs(low, high)
    lx, ly = x.astype(L), y.astype(L)
    d = np.log(ly / lx)
    with np.errstate(invalid="ignore", divide="ignore"):
        want = np.where(d == 0, 1, d / np.sinh(d) if inverse else np.tanh(d / 2) / (d / 2))
    limit = 2 * 0.36 * 2.0 ** -53 + 2.0 ** -53  # and the rounding of the result
    got = factors(inverse, x, y)
    far = np.abs(d) > 7.9 * np.log(2)
    # beyond: words of the smaller value keep 62 - 8 places and more, four roundings
    assert np.all(np.abs(got - want) <= limit + np.where(far, 2.0 ** -51 * want, 0))
    for f in (2 + inverse, 4 + inverse):  # each series in its whole range
        got = factors(f, x, y)
        inside = got >= 0
        assert np.all(np.abs(got - want)[inside] <= limit)
        if high <= (0.5 * SHORT if f < 4 else 0.98):
            assert np.all(inside)
