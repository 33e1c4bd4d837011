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


def _known_sums(ctx, rows, seed, mean):
    """A batch whose dL/dy are known to the bit (no weights, so y = 0): the
    gradients, the loss, dL/dy and the targets."""
    import torch

    mlp = R.Mlp(ctx, seed=11)
    mlp.set_params(np.zeros(R.MLP_NPARAM, dtype=np.float32))
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    t = torch.zeros((rows, 288), device="cuda")
    t[:, :280] = torch.randn((rows, 280), generator=g, device="cuda") + mean
    x = torch.zeros((rows, 16), dtype=torch.bfloat16, device="cuda")
    grad = torch.zeros(R.MLP_NPARAM, dtype=torch.float32, device="cuda")
    loss = torch.zeros(1, dtype=torch.float32, device="cuda")
    mlp.gradients(rows, x, t, grad, loss)
    scale = torch.tensor(1.0, device="cuda") / (torch.tensor(float(rows), device="cuda") * torch.tensor(280.0, device="cuda"))
    dy = ((2.0 * (0.0 - t[:, :280])) * scale).to(torch.bfloat16).to(torch.float32)
    torch.cuda.synchronize()
    mlp.close()
    return M.unpack(grad.cpu().numpy().astype(np.float64)), loss.double().item(), dy, t[:, :280]


def _rms(a, ref):
    return float(np.sqrt(((a - ref) ** 2).sum() / (ref ** 2).sum()))


@pytest.mark.parametrize("rows", [4096, 16384, 65536])
def test_bias_sums_are_as_exact_as_sums_of_256_row_slabs(ctx, rows):
    """Against fp64: the rms error over eight batches is at most a tenth above that
    of fp32 sums over slabs of 256 rows (eight lanes of 32 rows, the lanes in turn)
    added to the total one after another."""
    err, ref = [], []
    for seed in range(8):
        G, _, dy, _ = _known_sums(ctx, rows, seed, float(seed & 1))
        exact = dy.double().sum(0).cpu().numpy()
        v = dy.reshape(rows // 256, 32, 8, 280)
        lanes = v[:, 0].clone()
        for i in range(1, 32):
            lanes += v[:, i]
        slabs = lanes[:, 0].clone()
        for i in range(1, 8):
            slabs += lanes[:, i]
        slabs = slabs.cpu().numpy()
        total = np.zeros(280, dtype=np.float32)
        for s in slabs:
            total = total + s
        err.append(_rms(G["b4"][:280], exact))
        ref.append(_rms(total.astype(np.float64), exact))
    rms = lambda e: np.sqrt(np.mean(np.square(e)))
    assert rms(err) <= 1.1 * rms(ref), (rms(err), rms(ref))


@pytest.mark.parametrize("rows", [8, 72, 4104, 65536, 262144])
def test_loss_of_large_batches(ctx, rows):
    """Against fp64 from the same targets: 2^-24 a rounding, at most 16 sums of a
    thread, 12 of a block and its parts' 20 + 10 (20,480 parts, eight sums of 128
    threads) one after another, all of one sign; and the same in a second call."""
    for seed in range(4):
        _, loss, _, t = _known_sums(ctx, rows, seed, 0.5 * seed)
        exact = (t.double() ** 2).sum().item() / (rows * 280.0)
        # each term w e e scale: three roundings, and that of the scale
        assert abs(loss - exact) <= (16 + 12 + 30 + 4) * 2.0 ** -24 * exact, (loss, exact)
        assert abs(loss - exact) <= 6e-7 * exact, (loss, exact)  # ten roundings: what such sums are off in practice
        assert _known_sums(ctx, rows, seed, 0.5 * seed)[1] == loss
