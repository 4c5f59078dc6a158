"""A cell's results are the same bits whatever holds it: FP64 cells in shared memory and in global memory on clusters
(a CUDA-graph plan has no clusters; a plan of many tiles has none either), alone and among others of other sizes, cells
of at most ten nodes among cut ones, and FP32 cells whose place in the tile pairs their nodes with other cells'."""

import numpy as np
import pytest

from braincell_gb300 import workloads as W
from braincell_gb300.runtime import Plan

pytestmark = pytest.mark.gpu

DT = 0.025
STATES = ("V", "CaL_p", "CaL_q", "HCN_p", "Na_p", "KDR_p")


def _run(descs, precision, **kw):
    p = Plan(W.descs_to_batch(descs), precision=precision, record_every=3, **kw)
    for n in (400, 1, 99):  # past the first spikes
        p.run(n, DT)
    out = {k: p.state(k) for k in STATES}, p.traces(), p.info["n_smem_tiles"], p.cell_ncv()
    p.close()
    return out


@pytest.mark.parametrize("n_cells,lo,hi,tile", [(1, 505, 515, 0), (1, 1900, 2000, 0), (40, 3, 90, 800), (7, 300, 900, 2500),
                                                (5, 400, 2000, 0), (60, 50, 2000, 2500)])
def test_f64_clusters_give_the_bits_of_shared_memory_tiles(native_lib, cuda_device, n_cells, lo, hi, tile):
    descs = W.uneven(n_cells, n_range=(lo, hi))
    a, b = (_run(descs, "f64", tile_nodes=tile, use_graph=g) for g in (False, True))
    assert a[2] < b[2]  # the first plan's tiles did move
    for k in STATES:
        np.testing.assert_array_equal(a[0][k], b[0][k], err_msg=k)
    np.testing.assert_array_equal(a[1], b[1])


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("lo,hi", [(3, 9), (60, 90), (600, 900)])
def test_a_cell_alone_and_among_others(native_lib, cuda_device, precision, lo, hi):
    cell = W.uneven(1, n_range=(lo, hi), seed=11)
    alone = _run(cell, precision)
    # small and large mates, enough of the largest size that no tile is on a cluster
    for mates, kw in ((W.uneven(30, n_range=(3, 9)) + W.uneven(9, n_range=(40, 300)), {}),
                      (W.uneven(200, n_range=(600, 900)), {}), (W.uneven(9, n_range=(3, 200)), dict(tile_nodes=333))):
        for at in (0, len(mates) // 2):
            got = _run(mates[:at] + cell + mates[at:], precision, **kw)
            o = int(got[3][:at].sum())
            for k in STATES:
                np.testing.assert_array_equal(got[0][k][o:o + alone[3][0]], alone[0][k], err_msg=f"{k} {len(mates)} {at}")
