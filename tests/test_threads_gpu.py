"""Plans of different shared-memory sizes run from several host threads, each on a stream of its own: every launch
succeeds and the results are those of the plans run one after another.  Shared-memory tiles, and global-memory tiles
on clusters whose separators take shared memory."""

import threading

import numpy as np
import pytest

from braincell_gb300 import workloads as W
from braincell_gb300.runtime import Plan

pytestmark = pytest.mark.gpu

DT = 0.025
STEPS = 1500  # launches of one step each


def _plans(kind):
    if kind == "shared":
        batches = [W.uneven(20), W.small(1), W.uneven(2, n_range=(300, 400))]
    else:
        batches = [W.large(1), W.large(1, n_range=(6000, 6400), n_branches=60)]
    return [Plan(W.descs_to_batch(b), record_every=0) for b in batches]


@pytest.mark.parametrize("kind", ["shared", "global"])
def test_plans_run_from_several_threads(native_lib, cuda_device, kind):
    torch = pytest.importorskip("torch")
    alone = []
    for p in _plans(kind):
        p.run(STEPS, DT)
        alone.append(p.state("V"))
        p.close()
    plans = _plans(kind)
    errors = []

    def work(p, stream):
        try:
            for _ in range(STEPS):
                p.run(1, DT, stream=stream.cuda_stream, check=False)
            p.check(stream=stream.cuda_stream)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    streams = [torch.cuda.Stream() for _ in plans]
    threads = [threading.Thread(target=work, args=a) for a in zip(plans, streams)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for p, want in zip(plans, alone):
        np.testing.assert_array_equal(p.state("V"), want)
        p.close()
