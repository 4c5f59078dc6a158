"""Calcium shells with long time constants, up to one that never decays (tau infinite: Ci only
integrates its drive), against the float64 oracle: packed tiles, global-memory tiles and lane tiles.

FP64: 1e-8 mV and 1e-9 of Ci, as in the parity tests; FP32: 1e-3 mV, and 1e-5 of Ci, which a gain
that has lost its bits to a denormal quotient misses."""

from dataclasses import replace

import numpy as np
import pytest

from braincell_gb300 import workloads as W
from braincell_gb300.runtime import Plan
from oracle.staggered import OracleCell

pytestmark = pytest.mark.gpu

DT = 0.025


def _desc(tau):
    d = W.large(1, n_range=(60, 70), n_branches=6, n_pulses=8, duration=4.0)[0]
    return replace(d, ions_dend=[("CalciumDetailed", {"C_rest": 1e-4, "tau": tau, "d": 0.5, "Ci_initializer": 5e-5})])


@pytest.mark.parametrize("tau", [10.0, 1e6, 1e37, float("inf")])
@pytest.mark.parametrize("precision,tol_v,tol_ca", [("f64", 1e-8, 1e-9), ("f32", 1e-3, 1e-5)])
@pytest.mark.parametrize("lane", [0, 200])
def test_long_time_constants_match_the_oracle(native_lib, cuda_device, tau, precision, tol_v, tol_ca, lane):
    d = _desc(tau)
    p = Plan(W.descs_to_batch([d]), precision=precision, record_every=0, lane_cell_nodes=lane, device=cuda_device)
    n = 160
    p.run(n, DT)
    v, ci = p.state("V"), p.state("Ci")
    p.close()
    oc = OracleCell(W.desc_to_cell(d))
    oc.run(DT, n)
    has = np.isfinite(ci)
    ref = np.asarray(oc.Ci).reshape(-1)[oc.cv_mid][has]
    assert np.abs(ref - 5e-5).max() > 1e-6  # the drive has moved it
    assert np.abs(v - oc.V[0]).max() <= tol_v
    np.testing.assert_allclose(ci[has], ref, rtol=tol_ca, atol=0)
