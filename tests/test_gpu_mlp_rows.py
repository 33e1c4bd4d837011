"""Gradients of the training kernels over batch sizes around the row splits of
the weight gradients (256 rows each) and the 32-row tiles."""
import numpy as np
import pytest

from brams_gb300 import rrtmg_lw as R
from test_gpu_mlp import M, _dev_bf16, _rand_batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [8, 40, 264, 520, 2056])
def test_gradients_match_cpu_oracle(ctx, rows):
    """The bounds of the 256-row batch: bf16 activations, 1e-4 of the loss and
    2e-2 of each parameter block's largest gradient."""
    import torch

    mlp = R.Mlp(ctx, seed=11)
    p, _ = mlp.params()
    x, t = _rand_batch(rows, 5)
    td = torch.from_numpy(t).cuda()
    td[:, 280:] = float("nan")  # the padding is not read
    grad = torch.zeros(R.MLP_NPARAM, dtype=torch.float32, device="cuda")
    loss = torch.zeros(1, dtype=torch.float32, device="cuda")
    mlp.gradients(rows, _dev_bf16(x), td, grad, loss)
    torch.cuda.synchronize()
    l_ref, g_ref = M.forward_backward(p, x, t, emulate=True)
    assert abs(loss.item() - l_ref) <= 1e-4 * l_ref
    G, Gr = M.unpack(grad.cpu().numpy().astype(np.float64)), M.unpack(g_ref)
    for k in G:
        assert np.abs(G[k] - Gr[k]).max() <= 2e-2 * np.abs(Gr[k]).max() + 1e-12, k
