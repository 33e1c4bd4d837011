"""The transfer with and without the fluxes' temperature derivatives (their sums
are other code): one result in every launch shape and on every source of gas optics."""
import numpy as np
import pytest

from brams_gb300 import rrtmg_lw as R
from brams_gb300 import surrogate as S
from test_gpu_capture import NLAY, Batch, Dropin, Nomcica

pytestmark = pytest.mark.gpu

OFF = slice(7, 90)  # learned: these columns are wholly off the network


def _run(ctx, kind, c, nlay, idrv):
    import torch

    outs = [k for k in R.OUT_ORDER if idrv or not k.startswith("du")]
    for k in outs:
        c.d[k].zero_()
    if kind in ("batch", "learned"):
        d = R.grid_desc(c.n, nlay, c.d, icld=3, idrv=idrv, cloud_mode=R.CLOUD_FUSED, seed0=9)
        if kind == "learned":
            ctx.net.batch([d])
        else:
            ctx.rrtmg_lw_batch_device([d])
    elif kind == "dropin":
        ctx.rrtmg_lw_device(c.n, nlay, c.d, idrv=idrv)
    else:
        ctx.rrtmg_lw_nomcica_device(c.n, nlay, c.d, icld=1 if kind == "random" else 2, idrv=idrv)
    torch.cuda.synchronize()
    return {k: c.d[k].cpu().numpy().copy() for k in outs}


@pytest.mark.parametrize("idrv", [0, 1])
@pytest.mark.parametrize("nlay", [NLAY, NLAY - 1])
@pytest.mark.parametrize("kind", ["batch", "learned", "dropin", "random", "maxran"])
def test_every_launch_shape_gives_the_same_bits(kind, nlay, idrv):
    ctx = R.Context()
    cls = {"batch": Batch, "learned": Batch, "dropin": Dropin, "random": Nomcica, "maxran": Nomcica}[kind]
    c = cls(ctx, 170)
    c.d["emis"] = c.d["emis"] * 0.7  # a reflecting surface
    plain = None
    if kind == "learned":
        ctx.net = S.load(ctx)
        c.d["tlay"][:, OFF] += 200.0
        plain = _run(ctx, "batch", c, nlay, idrv)
    ref = None
    for v in range(ctx.num_variants()):
        for k in range(4):
            ctx.set_tuning(nlay, v, 1 + v % 2, kind=k)
        got = _run(ctx, kind, c, nlay, idrv)
        ref = ref or got
        assert got["uflx"].max() > 100.0
        for k in got:
            assert np.isfinite(got[k]).all() and np.array_equal(got[k], ref[k]), (k, v)
            if plain:
                assert np.array_equal(got[k][:, OFF], plain[k][:, OFF]), (k, v)
    assert ctx.sync_status() == 0
    if kind == "learned":
        ctx.net.close()
    ctx.close()
