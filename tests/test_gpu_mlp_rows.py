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


def test_one_accumulator_adds_at_most_2048_rows(ctx):
    """262,144 rows of one dL/dy and a first one 2^26 times as large: what an fp32
    accumulator that holds the first adds of the others is lost, 2,047 of them at
    most.  Adding up the blocks' sums (16 products are added at a time, 128 or more
    blocks) may lose a further 8 of the unit each.  Only b3 is nonzero, so that
    act3 = 32 and the last layer's gradient is 32 times the sum."""
    import torch

    rows, big = 262144, 2.0 ** 26
    mlp = R.Mlp(ctx, seed=11)
    d = {k: np.zeros(s) for k, s in M.SHAPES.items()}
    d["b3"][:] = 32.0
    mlp.set_params(M.pack(d).astype(np.float32))
    t = torch.zeros((rows, 288), device="cuda")
    t[:, :280] = -1.0
    t[0, :280] = -big
    x = torch.zeros((rows, 16), dtype=torch.bfloat16, device="cuda")
    grad = torch.zeros(R.MLP_NPARAM, dtype=torch.float32, device="cuda")
    loss = torch.zeros(1, dtype=torch.float32, device="cuda")
    mlp.gradients(rows, x, t, grad, loss)
    torch.cuda.synchronize()
    scale = np.float32(1.0) / (np.float32(rows) * np.float32(280.0))
    unit = float(M.bf16(np.array([np.float32(2.0) * scale]))[0])
    G = M.unpack(grad.cpu().numpy().astype(np.float64))
    exact = big + rows - 1
    for got in (G["b4"][:280] / unit, G["W4"][:, :280] / (32.0 * unit)):
        assert np.abs(got - exact).max() <= 2047 + 8 * 200, np.abs(got - exact).max()
