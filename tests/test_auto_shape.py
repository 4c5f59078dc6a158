"""Automatic tile shapes (``tile_nodes`` and ``threads_per_tile`` 0): two tiles to an SM for small
populations, the size that ran best for large ones; explicit values stand.  CPU (dry-run plans, which
count 152 SMs)."""

import numpy as np
import pytest

from braincell_gb300 import workloads as W
from braincell_gb300.runtime import Plan


@pytest.mark.parametrize("n,precision", [(1, "f32"), (16, "f32"), (700, "f32"), (16, "f64"), (3000, "f64")])
def test_small_cells_spread_over_the_gpu(native_lib, n, precision):
    p = Plan(W.descs_to_batch(W.small(n)), precision=precision, dry_run=True)
    nodes = 129 * n
    want = min(max(-(-nodes // 304), 128), 1250 if precision == "f64" else 2500)
    assert p.info["tile_nodes"] == want
    st = p.tile_stats()
    # whole cells: a tile holds as many as fit its budget, at least one
    assert p.info["n_tiles"] == -(-n // max(1, want // 129))
    assert st[:, 0].sum() == nodes
    T = p.info["threads_per_tile"]
    assert T % 32 == 0 and T == min(512, -(-(want // 2) // 32) * 32 + 32)


def test_explicit_shapes_stand(native_lib):
    p = Plan(W.descs_to_batch(W.small(40)), dry_run=True, tile_nodes=1000, threads_per_tile=64)
    assert p.info["tile_nodes"] == 1000 and p.info["threads_per_tile"] == 64
    assert np.all(p.tile_stats()[:, 0] <= 1000) and p.info["n_tiles"] == 6
