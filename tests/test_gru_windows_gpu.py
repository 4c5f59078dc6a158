"""GRU training kernels at the sizes where their staging changes form: windows around the 32-step
chunk, ragged batches, an offset window, and input buffers on 4-byte boundaries (no vector access).

The forward is causal and every sequence is its own, so the outputs of a short window or a small
batch are the leading part of those of a longer and larger one, bit for bit, whatever the staging:
no tolerance is needed.  The gradient has the bound of its own parity test.
"""

import numpy as np
import pytest

from oracle import gru as G

pytestmark = pytest.mark.gpu

N_MAX, T_MAX, T0 = 33, 97, 3


def _trainer(n, T, shift, device):
    import torch

    from braincell_gb300.gru import GRUTrainer

    rng = np.random.default_rng(19)
    x = rng.normal(size=(N_MAX, T_MAX + T0, G.X)).astype(np.float32)[:n, : T + T0]
    y = rng.normal(scale=0.5, size=(N_MAX, T_MAX + T0)).astype(np.float32)[:n, : T + T0]
    theta = G.init_params(7, scale=2.0).astype(np.float32)
    tr = GRUTrainer(np.ascontiguousarray(x), np.ascontiguousarray(y), theta, batch=n, window=T, device=device)
    if shift:  # the same buffers, 4 bytes on
        for name in ("x", "h", "acts", "y"):
            t = getattr(tr, name)
            buf = torch.empty(t.numel() + 4, dtype=torch.float32, device=t.device)
            view = buf[1:1 + t.numel()].view(t.shape)
            view.copy_(t)
            assert view.data_ptr() % 8 == 4
            setattr(tr, name, view)
    return x, y, theta, tr


@pytest.mark.parametrize("n,T", [(1, 1), (16, 31), (17, 32), (5, 33), (33, 64), (3, 65)])
@pytest.mark.parametrize("shift", [0, 1], ids=["aligned", "odd"])
def test_windows(native_lib, cuda_device, n, T, shift):
    full = _trainer(N_MAX, T_MAX, 0, cuda_device)[3].gradient(np.arange(N_MAX), T0, T_MAX)[2]
    x, y, theta, tr = _trainer(n, T, shift, cuda_device)
    loss, g, yout = tr.gradient(np.arange(n), T0, T)
    np.testing.assert_array_equal(yout, full[:n, :T])
    xs, ys = x[:, T0:].astype(np.float64), y[:, T0:].astype(np.float64)
    # FP64 sum of the FP32 outputs' squared errors: order and the final rounding only
    np.testing.assert_allclose(loss, np.mean((yout.astype(np.float64) - ys) ** 2), rtol=1e-6)
    ref, _, cache = G.forward(theta.astype(np.float64), xs, np.zeros((n, G.H)), quantize=True)
    gref = G.backward(theta.astype(np.float64), xs, ys, ref, cache, quantize=True)
    assert np.linalg.norm(g - gref) / np.linalg.norm(gref) < 1e-2
