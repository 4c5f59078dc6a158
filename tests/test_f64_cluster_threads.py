"""FP64 plans whose tiles move to clusters of CTAs keep the CTA size they were given.  CPU (dry-run plans): a tile's
length estimate, the walks of its busiest warp, shows the size its schedule was made for."""

import pytest

from braincell_gb300 import workloads as W
from braincell_gb300.runtime import Plan


def _plan(**kw):
    p = Plan(W.descs_to_batch(W.uneven(6, n_range=(600, 900))), precision="f64", dry_run=True, **kw)
    st = p.tile_stats()
    assert (st[:, 4] == 2).all() != bool(kw.get("use_graph"))
    return p.info["threads_per_tile"], st[:, 3]


@pytest.mark.parametrize("tile,key", [(2500, "threads_per_tile"), (64, "threads_big")])
def test_given_sizes_are_kept(native_lib, tile, key):
    small, s64 = _plan(tile_nodes=tile, **{key: 64})
    large, s512 = _plan(tile_nodes=tile, **{key: 512})
    assert (small, large) == (64, 512)
    assert (s64 > s512).all()
    # the same schedule as with the size given for global-memory tiles, which comes first where both are given
    t, s = _plan(tile_nodes=tile, threads_global=64)
    assert t == 64 and (s == s64).all()
    t, s = _plan(tile_nodes=tile, threads_global=512, **{key: 64})
    assert t == 512 and (s == s512).all()


def test_automatic_size(native_lib):
    t, s = _plan(tile_nodes=2500)
    assert t == 512 and (s == _plan(tile_nodes=2500, threads_per_tile=512)[1]).all()
