"""The tree solve at the shapes where its segments and separators change form: unbranched cells
(the root is the middle of the run), long runs cut into pieces, many branches at one point,
branches on both ends of the soma, and packed tiles that mix them.  FP64 kernels against the
float64 oracle at 1e-8 mV, as in the parity tests; FP32 against the same at 1e-3 mV."""

import numpy as np
import pytest

from braincell_gb300 import Branch, Cell, Morphology
from braincell_gb300 import workloads as W
from braincell_gb300.batch import concat_batches, lower_cell
from braincell_gb300.mech import AllRegion, CableProperty, Channel, CurrentClamp, CVPerBranchList, RootLocation, StateProbe
from braincell_gb300.runtime import Plan
from oracle.staggered import OracleCell

pytestmark = pytest.mark.gpu

DT = 0.025
# (parent, parent_x, compartments) per branch; branch 0 is the soma
SHAPES = {
    "one": [(-1, 0.0, 1)],
    "run_2": [(-1, 0.0, 2)],
    "run_3_1": [(-1, 0.0, 3), (0, 1.0, 1)],
    "run_500": [(-1, 0.0, 1), (0, 1.0, 500)],
    "star_9": [(-1, 0.0, 1)] + [(0, 1.0, n) for n in (1, 2, 3, 4, 5, 8, 9, 33, 40)],
    "both_ends": [(-1, 0.0, 3), (0, 0.0, 4), (0, 0.0, 7), (0, 1.0, 12), (0, 1.0, 1), (3, 1.0, 5), (3, 1.0, 64)],
    "comb": [(-1, 0.0, 1)] + [(2 * (k // 2), 1.0, 1 + k % 5) for k in range(24)],
}


def _cell(shape):
    m = Morphology.from_root(Branch.from_lengths(lengths=[20.0], radii=[10.0, 9.0], type="soma"), name="soma")
    for k, (par, x, n) in enumerate(SHAPES[shape][1:], 1):
        br = Branch.from_lengths(lengths=[7.0 * n + k], radii=[1.0 + 0.05 * k, 0.4], type="basal_dendrite")
        m.attach(parent=par, parent_x=x, child_branch=br, child_name=f"b{k}")
    c = Cell(m, cv_policy=CVPerBranchList(tuple(n for _, _, n in SHAPES[shape])))
    c.paint(AllRegion(), CableProperty(), Channel("IL", g_max=0.3, E=-70.0), Channel("CaL_IS2008", g_max=2.0),
            Channel("HCN_HM1992", g_max=0.02, E=-43.0))
    c.place(RootLocation(0.5), CurrentClamp(delay=0.5, durations=6.0, amplitudes=0.4))
    c.place(RootLocation(0.5), StateProbe())
    return c


@pytest.mark.parametrize("lane_nodes", [1, 10, 4000])
@pytest.mark.parametrize("precision,tol", [("f64", 1e-8), ("f32", 1e-3)])
def test_segment_shapes_match_the_oracle(native_lib, cuda_device, precision, tol, lane_nodes):
    cells = [_cell(s) for s in SHAPES]
    n = 300
    p = Plan(concat_batches([lower_cell(c) for c in cells]), precision=precision, tile_nodes=1000, threads_per_tile=96,
             lane_nodes=lane_nodes, device=cuda_device)
    p.run(n, DT)
    V = p.state("V")
    off = 0
    for name, c in zip(SHAPES, cells):
        oc = OracleCell(c)
        oc.run(DT, n)
        got = V[off:off + oc.V.shape[1]]
        assert np.abs(got - oc.V[0]).max() <= tol, name
        off += oc.V.shape[1]
    assert off == V.size


@pytest.mark.parametrize("n_cells", [1, 3, 20])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_clusters_do_not_change_a_global_memory_cell(native_lib, cuda_device, n_cells, precision):
    # cells too large for shared memory run on clusters of CTAs when they are few; a CUDA-graph
    # plan runs the same tiles on one CTA each: bit-identical
    descs = W.large(n_cells, n_range=(6000, 6400), n_branches=60, n_pulses=40, duration=4.0)
    out = []
    for use_graph in (False, True):
        p = Plan(W.descs_to_batch(descs), precision=precision, record_every=4, use_graph=use_graph, device=cuda_device)
        assert (p.tile_stats()[:, 4] == 2).any()
        for n in (60, 1, 39):
            p.run(n, DT)
        out.append((p.state("V"), p.state("Ci"), p.traces()))
        p.close()
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
