"""``set_pulse_amps`` and the time step: the amplitudes set last hold after the pulse records are made again for another
dt (after a reset), set before the first run or between runs, equal to a plan that was built with them.  Bits equal:
the records are the same numbers."""

from dataclasses import replace

import numpy as np
import pytest

from braincell_gb300 import workloads as W
from braincell_gb300.runtime import Plan

pytestmark = pytest.mark.gpu


def _descs(amps):
    out = []
    for k, d in enumerate(W.uneven(3, n_range=(20, 60))):
        mid = (1, 0.5, 0.5, 2.0)
        out.append(replace(d, pulses=[(0, 0.5, 0.2, 3.0, amps[2 * k]), (*mid, amps[2 * k + 1])]))
    return out


def _reference(amps, dt, n):
    p = Plan(W.descs_to_batch(_descs(amps)), precision="f64", record_every=0)
    p.run(n, dt)
    v = p.state("V")
    p.close()
    return v


@pytest.mark.parametrize("first", ["before any run", "after a run"])
def test_amplitudes_survive_a_new_time_step(native_lib, cuda_device, first):
    a = np.array([0.1, 0.2, 0.3, 0.05, 0.15, 0.25])
    b = np.array([0.4, -0.1, 0.0, 0.35, 0.22, 0.11])
    p = Plan(W.descs_to_batch(_descs(a)), precision="f64", record_every=0)
    if first == "after a run":
        p.run(50, 0.025)
        p.reset()
    p.set_pulse_amps(b)
    for dt, n in ((0.025, 120), (0.0125, 200), (0.05, 60)):
        p.run(n, dt)
        np.testing.assert_array_equal(p.state("V"), _reference(b, dt, n), err_msg=f"dt {dt}")
        p.reset()
    p.set_pulse_amps(a)  # and back, at the dt of the last run and at another
    for dt, n in ((0.05, 60), (0.025, 120)):
        p.run(n, dt)
        np.testing.assert_array_equal(p.state("V"), _reference(a, dt, n), err_msg=f"dt {dt}")
        p.reset()
    p.close()
