"""The pair pressure of the moist and rainy two-point fluxes is a quotient with one rounding, not a
product with a rounded reciprocal: where numerator and denominator are equal integers it is exactly 1
(y fl(1/y) is not for 49, 98, 103, ...).  The pair functions are compiled for the host."""
import ctypes
import os
import shutil
import subprocess

import numpy as np

from test_int_math import CSRC

HARNESS = r"""
#include "phys_moist_2d.cuh"
#include "phys_rainy_2d.cuh"
using namespace tag;
namespace tag { void set_last_error(const std::string&) {} }
extern "C" void pressures(long n, const double* y, double* moist, double* rainy) {
  PhysMoist2D::Params P{};
  P.R_d = 1.0;
  for (long i = 0; i < n; ++i) {
    double q[16] = {}, Fa[9], Fb[9];
    q[0] = q[6] = 0.5 * y[i];  // dry density and 1/T, halved
    q[5] = 1.0;
    PhysMoist2D::volume_pair(P, q, q, 0.0, 1.0, Fa, Fb);
    moist[i] = Fa[2];
    double r[16] = {};
    r[0] = 0.5 * y[i];
    r[7] = 0.5 * RainyConst::R_d * y[i];
    r[6] = 1.0;
    PhysRainy2D::volume_pair(PhysRainy2D::Params{}, r, r, 0.0, 1.0, Fa, Fb);
    rainy[i] = Fa[4];
  }
}
"""


def test_pair_pressure_is_a_quotient(tmp_path):
    src, lib = tmp_path / "harness.cu", tmp_path / "harness.so"
    src.write_text(HARNESS)
    home = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    nvcc = shutil.which("nvcc") or os.path.join(home, "bin", "nvcc")
    subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_103a,code=sm_103a", "-shared",
                    "-Xcompiler", "-fPIC", "-I", CSRC, str(src), "-o", str(lib)], check=True)
    fn = ctypes.CDLL(str(lib)).pressures
    dp = np.ctypeslib.ndpointer(np.float64, flags="C")
    fn.argtypes = [ctypes.c_long, dp, dp, dp]
    y = np.arange(1.0, 2001.0)
    assert np.sum(y * (1 / y) != 1) > 50
    moist, rainy = np.zeros_like(y), np.zeros_like(y)
    fn(y.size, y, moist, rainy)
    assert np.all(moist == 1) and np.all(rainy == 1)
