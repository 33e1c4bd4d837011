"""Caller sub-columns through the cells' kernel: ragged grids in one batch with
an odd number of columns, several passes, arrays on 8-byte boundaries, and
the water paths around cldprmc's 1e-20."""
import numpy as np
import pytest

import pyoracle
from brams_gb300 import rrtmg_lw as R
from brams_gb300 import surrogate as S
from brams_gb300.profiles import ProfileSpec, make_state

pytestmark = pytest.mark.gpu

FLUX_TOL, HR_TOL = 0.05, 0.01  # the solver's parity tolerances (W m-2, K/day)
CELLS = ("cldfmcl", "ciwpmcl", "clwpmcl", "taucmcl")


def _cells(mc, shift=0):
    """The (140, ncol, nlay) arrays on the device, `shift` doubles past a 16-byte boundary."""
    import torch

    out = {}
    for k in CELLS:
        v = np.ascontiguousarray(mc[k].T).ravel()
        b = torch.zeros(v.size + 2, dtype=torch.float64, device="cuda")
        b[shift:shift + v.size] = torch.from_numpy(v)
        out[k] = b[shift:]
    return out


def _grid(st, mc, shift):
    g = S.DeviceGrid(st, pyoracle.cldprop_columns(st))
    g.d.update(_cells(mc, shift))
    desc = R.grid_desc(g.ncol, g.nlay, {**g.d, "reicmcl": g.d["rei"], "relqmcl": g.d["rel"]}, icld=3,
                       cloud_mode=R.CLOUD_SUBCOL)
    return g, desc


def _check(got, ref):
    for k in ("uflx", "dflx", "uflxc", "dflxc"):
        assert np.abs(got[k] - ref[k]).max() <= FLUX_TOL, k
    for k in ("hr", "hrc"):
        assert np.abs(got[k] - ref[k]).max() <= HR_TOL, k


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("shapes", [[(1, 38)], [(3, 45), (33, 38), (7, 60)], [(155, 45), (31, 128)], [(201, 7)]])
def test_ragged_batches_against_oracle(ctx, shapes, shift):
    import torch

    grids, descs, refs = [], [], []
    for i, (ncol, nlay) in enumerate(shapes):
        st = make_state(ProfileSpec(ncol=ncol, nlay=nlay, seed=800 + i, t_noise=4.0, cloud_prob=0.6))
        mc = pyoracle.mcica_per_column(st, pyoracle.cldprop_columns(st), icld=3, base_seed=40 + i)
        rs = np.random.default_rng(i)
        for k in ("ciwpmcl", "clwpmcl"):  # paths whose sum is below, at and above the threshold
            edge = rs.random(mc[k].shape) < 0.05
            mc[k] = np.asfortranarray(np.where(edge, rs.choice([0.0, 5e-21, 1e-20, 9.9e-21, 1e-300], mc[k].shape), mc[k]))
        g, d = _grid(st, mc, shift)
        grids.append(g)
        descs.append(d)
        refs.append(pyoracle.rrtmg_lw(st, mc, icld=3))
    ctx.rrtmg_lw_batch_device(descs)
    torch.cuda.synchronize()
    assert ctx.sync_status() == 0
    for g, ref in zip(grids, refs):
        _check(g.outputs(), ref)


def test_several_passes_repeat_their_columns(ctx):
    """131 columns of 128 layers, 121 times over (a pass holds about 6,000): every copy has the first one's bits."""
    import torch

    st = make_state(ProfileSpec(ncol=131, nlay=128, seed=9, t_noise=4.0, cloud_prob=0.6))
    mc = pyoracle.mcica_per_column(st, pyoracle.cldprop_columns(st), icld=3, base_seed=3)
    g, desc = _grid(st, mc, 0)
    ctx.rrtmg_lw_batch_device([desc])
    torch.cuda.synchronize()
    one = {k: v.copy() for k, v in g.outputs().items()}
    n = 121
    for k, v in list(g.d.items()):
        if k in CELLS:
            v = v[: 140 * 131 * 128].reshape(128, 131, 140)
            g.d[k] = v.repeat(1, n, 1).contiguous()
        elif v.shape[-1] == 131:
            g.d[k] = v.repeat(*([1] * (v.dim() - 1)), n).contiguous()
    g.ncol = n * 131
    desc = R.grid_desc(g.ncol, 128, {**g.d, "reicmcl": g.d["rei"], "relqmcl": g.d["rel"]}, icld=3,
                       cloud_mode=R.CLOUD_SUBCOL)
    ctx.rrtmg_lw_batch_device([desc])
    torch.cuda.synchronize()
    assert ctx.sync_status() == 0
    got = g.outputs()
    for k, v in one.items():
        assert np.array_equal(got[k].reshape(n, 131, -1), np.broadcast_to(v, (n,) + v.shape)), k
