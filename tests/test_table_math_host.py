"""The FP64 table-driven exponential and logarithm, on the host, against exact values (50 digits).

Bounds, in units u = 2^-53.  2^(y / 256): table entry 1 u, last rounding 1 u, polynomial 0.4 u.
ln x: table entry and last term 3 u, product with the exponent and sum 3 u of the result.
Needs nvcc (no GPU)."""

import ctypes as C
import decimal
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
DP = C.POINTER(C.c_double)
U = 2.0**-53
D = decimal.Decimal


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not available")
    out = str(tmp_path_factory.mktemp("table_math") / "libtable_math.so")
    subprocess.run([nvcc, "-x", "cu", "-shared", "-Xcompiler", "-fPIC", "-std=c++17", "-O2",
                    "-gencode=arch=compute_103a,code=sm_103a", os.path.join(HERE, "table_math_host.cu"), "-o", out],
                   check=True, capture_output=True, text=True)
    return C.CDLL(out)


def _call(fn, x):
    x = np.ascontiguousarray(x, dtype=np.float64)
    out = np.zeros_like(x)
    fn(x.ctypes.data_as(DP), x.size, out.ctypes.data_as(DP))
    return out


def _rel(got, want):
    with decimal.localcontext() as ctx:
        ctx.prec = 50
        return max(abs(float(D(float(g)) / w - 1)) for g, w in zip(got, want))


def test_exponential(lib):
    rng = np.random.default_rng(3)
    # every table entry, both edges of its interval, and random arguments up to 2^+-1000
    y = np.concatenate([np.arange(-300, 300), np.arange(-300, 300) + np.nextafter(0.5, 0),
                        rng.uniform(-2e4, 2e4, 1500), rng.uniform(-2.56e5, 2.56e5, 500)])
    with decimal.localcontext() as ctx:
        ctx.prec = 50
        want = [(D(float(t)) / 256 * D(2).ln()).exp() for t in y]
    assert _rel(_call(lib.bc_test_exp2_256, y), want) < 2.4 * U


def test_exponential_far_out(lib):
    got = _call(lib.bc_test_exp2_256, [3e5, 1e300, np.inf, -3e5, -1e300, -np.inf])
    assert np.isfinite(got).all() and (got[:3] > 1e303).all() and (got[3:] < 1e-303).all() and (got > 0).all()
    assert np.isnan(_call(lib.bc_test_bell, [np.nan])).all()


def test_linear_argument(lib):
    v = np.linspace(-150.0, 90.0, 1201)
    with decimal.localcontext() as ctx:
        ctx.prec = 50
        arg = [-(D(float(t)) + 59) / D(6.2) for t in v]
        want = [a.exp() for a in arg]
    # the product, the constant and their sum: 3 roundings of terms of at most 150 / 6.2 + 59 / 6.2
    assert _rel(_call(lib.bc_test_line, v), want) < (2.4 + 3 * 209 / 6.2) * U


def test_logarithm(lib):
    rng = np.random.default_rng(4)
    j = 1.0 + np.arange(256) / 256
    x = np.concatenate([j, np.nextafter(j, 0), j * 2.0**-13, np.exp(rng.uniform(-20, 10, 1500)),
                        np.exp(rng.uniform(-700, 700, 300)), [2.0**-1022, 1.7e308]])
    with decimal.localcontext() as ctx:
        ctx.prec = 50
        want = [D(float(t)).ln() for t in x]
    got = _call(lib.bc_test_ln, x)
    for g, w in zip(got, want):
        assert abs(D(float(g)) - w) < D(3 * U) + D(3 * U) * abs(w)


def test_logarithm_elsewhere(lib):
    with np.errstate(all="ignore"):
        x = np.array([0.0, -0.0, -1.0, 1e-310, np.inf, np.nan])
        np.testing.assert_array_equal(_call(lib.bc_test_ln, x), np.log(x))
