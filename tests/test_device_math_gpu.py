"""The device forms of the library's own arithmetic (``bc_mech.cuh``), compiled for sm_103a.

FP32, u = 2^-24 (half an ulp, relative):
- ``adiv(a, b)``, ``adiv_sum(a, b)``: the quotient's residual is exact but for its own rounding, and the correction is 2^-22 of the
  quotient, so what is left is the last rounding, 1 u, and 2^-44;
- ``over_exprel(c, x)`` = c x / (e^x - 1): the product 1 u, CUDA's expm1f 1 ulp = 2 u, the division 1 u;
- ``over_1pexp(c, x)`` = c / (1 + e^x): CUDA's expf 2 ulp = 4 u, the sum 1 u, the division 1 u.

FP64, u = 2^-53 (``ln_pos`` and ``exp2_256`` against exact values, as the host test has them):
- ``srcp(x)``: the estimate takes 24 bits of x (off by 2^-23 at most) and is CUDA's FP32 approximation of their
  reciprocal (1 ulp, 2^-23), so |e| = |1 - x r| <= 2^-22; the series r (1 + e + e^2) leaves e^3 = 2^-66 and the last
  rounding, 1 u.  CUDA's 1.0 / x is the correctly rounded one.
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
RCP, EXP2_256, LN, DIV, OVER_EXPREL, OVER_1PEXP, DIV_SUM = range(7)
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
    for fn in (DIV, DIV_SUM):
        x, y, q = _f32(lib, fn, a, b)
        assert np.max(np.abs(q / (x / y) - 1.0)) <= U32 * (1 + 2.0**-18)


def test_fp32_division_at_the_ends(lib):
    # rates of a gate far outside its range: a finite rate over an infinite sum is 0, as the IEEE quotient
    inf, nan = np.inf, np.nan
    a, b, q = _f32(lib, DIV_SUM, [0.0, 1.0, 1e30, 0.0, 1e-30, inf, nan, 1.0], [inf, inf, inf, 1e30, 1e38, inf, 1.0, nan])
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


def _relative_error(got, want):
    with decimal.localcontext() as ctx:
        ctx.prec = 50
        return max(abs(float(D(float(g)) / w - 1)) for g, w in zip(got, want))


def test_fp64_reciprocal(lib):
    rng = np.random.default_rng(2)
    ends = [1.0, np.nextafter(1.0, 2.0), np.nextafter(2.0, 1.0), np.nextafter(1.0, 0.0), 1.5, 4.0 / 3.0, 1.0 + 2.0**-23,
            1.0 + 2.0**-20, 2.0 - 2.0**-20, 1.0 - 2.0**-24]
    # mantissas of every leading pattern's ends, exponents over the whole range, 2^+-1008 among them
    x = np.concatenate([np.ldexp(rng.uniform(1.0, 2.0, 400_000), rng.integers(-1021, 1020, 400_000)),
                        np.outer(np.exp2(np.r_[-1008:1009:96, 0]), ends).ravel(), 1.0 + np.arange(4096) / 4096,
                        np.nextafter(1.0 + np.arange(4096) / 4096, 0.0)])
    x = np.concatenate([x, -x])
    got, want = _f64(lib, RCP, x), 1.0 / x
    near = np.abs(got - want) <= np.spacing(np.abs(want))
    assert near.all()
    # the correctly rounded value but where 1 / x lies within 2^-13 u of the middle of two numbers
    off = np.nonzero(got != want)[0]
    assert off.size <= 2.0**-11 * x.size
    for k in off:
        assert abs(Fraction(float(got[k])) * Fraction(float(x[k])) - 1) <= Fraction(U64) * (1 + Fraction(1, 4096))


def test_fp64_reciprocal_of_nan(lib):
    assert np.isnan(_f64(lib, RCP, [np.nan, -np.nan])).all()


def test_fp64_exponential(lib):
    rng = np.random.default_rng(3)
    y = np.concatenate([np.arange(-300, 300), np.arange(-300, 300) + np.nextafter(0.5, 0),
                        rng.uniform(-2e4, 2e4, 1500), rng.uniform(-2.56e5, 2.56e5, 500)])
    with decimal.localcontext() as ctx:
        ctx.prec = 50
        want = [(D(float(t)) / 256 * D(2).ln()).exp() for t in y]
    assert _relative_error(_f64(lib, EXP2_256, y), want) < 2.4 * U64
    far = _f64(lib, EXP2_256, [3e5, 1e300, np.inf, -3e5, -1e300, -np.inf])
    assert np.isfinite(far).all() and (far[:3] > 1e303).all() and (far[3:] < 1e-303).all() and (far > 0).all()


def test_fp64_logarithm(lib):
    rng = np.random.default_rng(4)
    j = 1.0 + np.arange(256) / 256
    x = np.concatenate([j, np.nextafter(j, 0), j * 2.0**-13, np.exp(rng.uniform(-20, 10, 1500)),
                        np.exp(rng.uniform(-700, 700, 300)), [2.0**-1022, 1.7e308]])
    with decimal.localcontext() as ctx:
        ctx.prec = 50
        want = [D(float(t)).ln() for t in x]
    for g, w in zip(_f64(lib, LN, x), want):
        assert abs(D(float(g)) - w) < D(3 * U64) + D(3 * U64) * abs(w)
    with np.errstate(all="ignore"):
        x = np.array([0.0, -0.0, -1.0, 1e-310, np.inf, np.nan])
        np.testing.assert_allclose(_f64(lib, LN, x), np.log(x), rtol=4 * U64, equal_nan=True)
