"""Tile budgets far above what shared memory holds: plans are made, and of tiles that fit.  CPU (dry-run plans)."""

import pytest

from braincell_gb300 import workloads as W
from braincell_gb300.runtime import Plan


def _cable(n):
    return W.CellDesc(parent=[-1, 0], length=[20.0, 5.0 * n], r_prox=[10.0, 1.0], r_dist=[10.0, 1.0], ncv=[1, n],
                      types=["soma", "dendrite"], channels_soma=[("IL", {})], channels_dend=[("IL", {})], probes=[])


@pytest.mark.parametrize("n,count,precision", [
    (1000, 3300, "f32"),  # 72,600 separators in all, more than a tile's indices count
    (1000, 40, "f64"),    # few tiles: on clusters, but not all cells on one
    (20000, 3, "f32"),    # cells that no shared memory holds
])
def test_a_huge_budget(native_lib, n, count, precision):
    p = Plan(W.descs_to_batch([_cable(n)] * count), precision=precision, dry_run=True, tile_nodes=1 << 23)
    st = p.tile_stats()
    total = p.info["n_nodes"]
    assert p.info["tile_nodes"] == 1 << 23 and st[:, 0].sum() == total
    per_node = 32 if precision == "f32" else 56  # bytes that every node takes of 227 KB
    assert st[:, 0].max() <= max(232448 // per_node, total // count)
    if n < 2000:
        assert p.info["n_tiles"] > 1 and (precision == "f64" or (st[:, 4] < 2).all())
