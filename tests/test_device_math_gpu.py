"""The device forms of the library's own arithmetic (``bc_mech.cuh``), compiled for sm_103a.

FP32, u = 2^-24 (half an ulp, relative):
- ``adiv(a, b)``: the quotient's residual is exact but for its own rounding, and the correction is 2^-22 of the
  quotient, so what is left is the last rounding, 1 u, and 2^-44;
- ``over_exprel(c, x)`` = c x / (e^x - 1): the product 1 u, CUDA's expm1f 1 ulp = 2 u, the division 1 u;
- ``over_1pexp(c, x)`` = c / (1 + e^x): CUDA's expf 2 ulp = 4 u, the sum 1 u, the division 1 u.

FP64, u = 2^-53 (``ln_pos`` and ``exp2_256`` against exact values, as the host test has them):
- ``srcp(x)``: the hardware estimate takes 20 bits of x and gives 20 bits, so |e| = |1 - x r| < 2^-18.5; the series
  r (1 + e + e^2) leaves e^3 < 2^-55.5 = 0.18 u, and the last rounding 1 u.
"""

import ctypes as C
import decimal
import os
import shutil
import subprocess
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
RCP, EXP2_256, LN, DIV, OVER_EXPREL, OVER_1PEXP = range(6)
U32, U64 = 2.0**-24, 2.0**-53
D = decimal.Decimal


@pytest.fixture(scope="module")
def lib(tmp_path_factory, cuda_device):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    out = str(tmp_path_factory.mktemp("device_math") / "libdevice_math.so")
    subprocess.run([nvcc, "-x", "cu", "-shared", "-Xcompiler", "-fPIC", "-std=c++17", "-O3", "--expt-relaxed-constexpr",
                    "-gencode=arch=compute_103a,code=sm_103a", os.path.join(HERE, "device_math.cu"), "-o", out],
                   check=True, capture_output=True, text=True)
    return C.CDLL(out)


def _f32(lib, fn, a, b):
    a, b = (np.ascontiguousarray(x, dtype=np.float32) for x in np.broadcast_arrays(np.float32(a), np.float32(b)))
    out = np.zeros_like(a)
    p = C.POINTER(C.c_float)
    assert lib.bc_test_device_f32(fn, a.ctypes.data_as(p), b.ctypes.data_as(p), a.size, out.ctypes.data_as(p)) == 0
    return a.astype(np.float64), b.astype(np.float64), out.astype(np.float64)


def _f64(lib, fn, x):
    x = np.ascontiguousarray(x, dtype=np.float64)
    out = np.zeros_like(x)
    p = C.POINTER(C.c_double)
    assert lib.bc_test_device_f64(fn, x.ctypes.data_as(p), x.size, out.ctypes.data_as(p)) == 0
    return out


def test_fp32_division(lib):
    rng = np.random.default_rng(1)
    n = 200_000
    a = rng.choice([-1.0, 1.0], n) * np.exp2(rng.uniform(-60, 60, n))
    b = rng.choice([-1.0, 1.0], n) * np.exp2(rng.uniform(-60, 60, n))
    a, b, q = _f32(lib, DIV, a, b)
    assert np.max(np.abs(q / (a / b) - 1.0)) <= U32 * (1 + 2.0**-18)


def test_fp32_division_at_the_ends(lib):
    # rates of a gate far outside its range: a finite rate over an infinite sum is 0, as the IEEE quotient
    inf, nan = np.inf, np.nan
    a, b, q = _f32(lib, DIV, [0.0, 1.0, 1e30, 0.0, 1e-30, inf, nan, 1.0], [inf, inf, inf, 1e30, 1e38, inf, 1.0, nan])
    np.testing.assert_array_equal(q[:4], 0.0)
    assert abs(q[4]) <= 1.2e-38  # below the normal numbers
    assert np.isnan(q[5:]).all()


def test_fp32_rate_forms(lib):
    x = np.concatenate([np.linspace(-100.0, 79.9, 20001), [0.0, 1e-35, -1e-35, 1e-7, -1e-7]])
    c, xs, got = _f32(lib, OVER_EXPREL, 1.28, x)
    with np.errstate(invalid="ignore", divide="ignore"):
        want = np.where(np.abs(xs) < 1e-30, c, c * xs / np.expm1(xs))
    assert np.max(np.abs(got / want - 1.0)) <= 4 * U32 * 1.01
    c, xs, got = _f32(lib, OVER_1PEXP, 4.0, x)
    assert np.max(np.abs(got * (1.0 + np.exp(xs)) / c - 1.0)) <= 6 * U32 * 1.01
    far = np.array([80.0, 100.0, 1e4, np.inf])
    for fn in (OVER_EXPREL, OVER_1PEXP):
        c, _, got = _f32(lib, fn, 4.0, far)
        assert (got >= 0).all() and (got <= 1e-31).all()
