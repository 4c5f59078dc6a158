"""FP32 cells of one-micrometre compartments against FP64.

Cylinders of radius 1 um, length 1 um: alpha = r / (2 R_a c_m L^2) = 5e4 / ms, alpha dt = 1,250.  A cell of at most ten
nodes is eliminated with plain diagonals, and a separator's row takes 1 - q - u and wE - wF: differences of numbers of
the order of alpha dt (or, times alpha dt, of 1), rounded to 2^-24.  An excess of the order of 1 is then off by up to
3 alpha dt 2^-24 (the two products and the difference), and the voltage, the sum of the increments, by that part of
the way it went.  Nodes inside segments take no difference."""

import numpy as np
import pytest

from braincell_gb300 import Branch, Cell, Morphology
from braincell_gb300.batch import lower_cell
from braincell_gb300.mech import AllRegion, CableProperty, Channel, CurrentClamp, CVPerBranchList, RootLocation, StateProbe
from braincell_gb300.runtime import Plan

pytestmark = pytest.mark.gpu

DT = 0.025
ALPHA_DT = 1e-4 / (2 * 100.0 * 1e-6 * 1e-8) * 1e-3 * DT
SHAPES = {
    "one": ([], []),
    "run_of_8": ([0], [7]),                       # 11 nodes: cut
    "y_of_9_nodes": ([0, 0, 0], [1] * 3),         # solved whole
    "run_of_10_nodes": ([0], [6]),                # solved whole
    "run_of_300": ([0], [299]),
    "branches_of_1": ([0] + [(i + 1) // 2 for i in range(1, 63)], [1] * 63),
    "branches_of_12": ([0, 0, 1, 1, 2, 2], [12] * 6),
    "run_of_5000": ([0], [4999]),
}


def _batch(parents, ncv):
    m = Morphology.from_root(Branch.from_lengths(lengths=[1.0], radii=[1.0, 1.0], type="soma"), name="soma")
    for k, (par, n) in enumerate(zip(parents, ncv), 1):
        m.attach(parent=par, parent_x=1.0, child_name=f"b{k}",
                 child_branch=Branch.from_lengths(lengths=[float(n)], radii=[1.0, 1.0], type="dendrite"))
    c = Cell(m, cv_policy=CVPerBranchList((1, *ncv)))
    c.paint(AllRegion(), CableProperty(), Channel("IL", g_max=0.3, E=-70.0), Channel("CaL_IS2008", g_max=0.5))
    c.place(RootLocation(0.5), CurrentClamp(delay=0.5, durations=100.0, amplitudes=2e-4 * (1 + sum(ncv)) ** 0.5))
    c.place(RootLocation(0.5), StateProbe())
    return lower_cell(c)


@pytest.mark.parametrize("shape", list(SHAPES))
def test_short_compartments(native_lib, cuda_device, shape):
    batch = _batch(*SHAPES[shape])
    tr, v = {}, {}
    for prec in ("f32", "f64"):
        p = Plan(batch, precision=prec, record_every=1, device=cuda_device)
        p.run(400, DT)
        tr[prec], v[prec] = p.traces(), p.state("V")
        p.close()
    way = np.abs(np.diff(tr["f64"], axis=1)).sum() + 1.0  # mV, by the clamped compartment
    bound = 3 * ALPHA_DT * 2.0**-24 * way
    assert np.abs(tr["f32"] - tr["f64"]).max() <= bound
    assert np.abs(v["f32"] - v["f64"]).max() <= bound
