"""The step's merged gate forms (steady state and -dt phi / tau without tau) and the decay series,
in FP64 on the host, against the rate structures that test_rates_host.py holds to the oracle, and
against expm1.  Needs nvcc (no GPU)."""

import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
DP = C.POINTER(C.c_double)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc is not available")
    out = str(tmp_path_factory.mktemp("step_rates") / "libstep_rates.so")
    subprocess.run([nvcc, "-x", "cu", "-shared", "-Xcompiler", "-fPIC", "-std=c++17", "-O2",
                    "-gencode=arch=compute_103a,code=sm_103a", os.path.join(HERE, "step_rates_host.cu"), "-o", out],
                   check=True, capture_output=True, text=True)
    return C.CDLL(out)


@pytest.mark.parametrize("which", range(5))
def test_step_forms_match_the_rate_structures(lib, which):
    # the branch point of CaT's q time constant (-80) and the bells' centres included
    v = np.concatenate([np.linspace(-150.0, 90.0, 2401), [-80.0, np.nextafter(-80.0, -81.0), -5.0, -40.0]])
    out = np.zeros((v.size, 4))
    assert lib.bc_test_step_rates(which, v.ctypes.data_as(DP), v.size, out.ctypes.data_as(DP)) == 0
    # a sum of at most five roundings and an exponential of an argument of up to 80 (its rounding times 80)
    np.testing.assert_allclose(out[:, :2], out[:, 2:], rtol=2e-14, atol=0)


def test_step_forms_stay_finite_far_out(lib):
    v = np.array([-1e4, -1e3, 1e3, 1e4])
    for which in range(5):
        out = np.zeros((v.size, 4))
        assert lib.bc_test_step_rates(which, v.ctypes.data_as(DP), v.size, out.ctypes.data_as(DP)) == 0
        assert np.isfinite(out[:, 0]).all() and (out[:, 0] >= 0).all() and (out[:, 0] <= 1).all()
        assert np.isfinite(out[:, 1]).all() and (out[:, 1] <= 0).all()


def test_decay_series_matches_expm1(lib):
    e = np.nextafter([0.015625, 0.125], 0.0)
    x = -np.concatenate([[0.0, 1e-300, 1e-9], np.geomspace(1e-12, 30.0, 3000), [0.015625, 0.125], e])
    out = np.zeros_like(x)
    lib.bc_test_decay(x.ctypes.data_as(DP), x.size, out.ctypes.data_as(DP))
    np.testing.assert_allclose(out, np.expm1(x), rtol=4e-16, atol=0)
