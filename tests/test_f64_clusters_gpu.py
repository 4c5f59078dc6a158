"""FP64 tiles on clusters of CTAs against the same plan in shared memory (a plan that runs as a CUDA graph has no
clusters): one cell and several to a tile, sizes either side of the rule, every state."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_cells,lo,hi,tile", [(1, 505, 515, 0), (1, 1900, 2000, 0), (40, 3, 90, 800), (7, 300, 900, 2500),
                                                (5, 400, 2000, 0)])
def test_matches_the_shared_memory_tiles(native_lib, cuda_device, n_cells, lo, hi, tile):
    from braincell_gb300 import workloads as W
    from braincell_gb300.runtime import Plan

    batch = W.descs_to_batch(W.uneven(n_cells, n_range=(lo, hi)))
    out = []
    for graph in (False, True):
        p = Plan(batch, precision="f64", tile_nodes=tile, record_every=2, use_graph=graph)
        p.run(40, 0.025)
        p.run(33, 0.025)
        out.append((p.info["n_smem_tiles"], p.traces(), {k: p.state(k) for k in ("V", "CaL_p", "Ci")}))
        p.close()
    assert out[0][0] < out[1][0]  # the rule took effect
    np.testing.assert_allclose(out[0][1], out[1][1], rtol=1e-11, atol=1e-11)
    for k, v in out[1][2].items():
        # the same operations on the same numbers, but for the order in which a separator's terms are summed
        np.testing.assert_allclose(out[0][2][k], v, rtol=1e-11, atol=1e-11, err_msg=k)
