"""The sub-column generator's draws and arrays bit for bit: column counts around
the fill's 4 and the draws' 32 columns, layer counts around its chunks of 16,
each overlap, and output arrays on 8-byte boundaries."""
import numpy as np
import pytest

import pyoracle
from brams_gb300.profiles import ProfileSpec, make_state
from test_gpu_cldprop_sw import _dev
from test_sw import _sw_band

pytestmark = pytest.mark.gpu

SUB = ("cldfmcl", "ciwpmcl", "clwpmcl", "taucmcl")


def _state(ncol, nlay, seed):
    st = make_state(ProfileSpec(ncol=ncol, nlay=nlay, seed=seed, cloud_prob=0.7))
    st["cldfrac"][0, :] = 1.0  # an overcast column
    st["alpha"] = np.asfortranarray(np.exp(-np.linspace(0.1, 2.0, nlay))[None, :] * np.ones((ncol, 1)))
    return st


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("ncol,nlay,icld", [(1, 1, 3), (3, 15, 3), (33, 16, 3), (37, 17, 3), (65, 33, 3), (5, 17, 1),
                                            (6, 33, 2), (2, 16, 4), (7, 5, 5)])
def test_longwave_sub_columns(ctx, ncol, nlay, icld, shift):
    import torch

    st = _state(ncol, nlay, 70 + ncol)
    tauc = pyoracle.cldprop_columns(st)
    d = {k: _dev(st[k]) for k in ("play", "cldfrac", "ciwp", "clwp", "rei", "rel", "alpha")}
    d["tauc"] = torch.from_numpy(np.ascontiguousarray(tauc.T)).cuda()
    n = 140 * ncol * nlay
    buf = {k: torch.full((n + 2,), -7.0, dtype=torch.float64, device="cuda") for k in SUB}
    d.update({k: v[shift:] for k, v in buf.items()})
    d["reicmcl"], d["relqmcl"] = torch.zeros_like(d["rei"]), torch.zeros_like(d["rel"])
    ctx.mcica_subcol_lw_device(ncol, nlay, d, icld=icld, permuteseed=-3, seed_per_column=True)
    torch.cuda.synchronize()
    for c in range(ncol):
        one = {k: np.asfortranarray(st[k][c:c + 1]) for k in ("play", "cldfrac", "ciwp", "clwp", "rei", "rel")}
        ref = pyoracle.mcica_subcol_lw(one, np.asfortranarray(tauc[:, c:c + 1]), icld, c - 3, 1,
                                       np.asfortranarray(st["alpha"][c:c + 1]) if icld >= 4 else None)
        for k in SUB:
            got = buf[k][shift:shift + n].cpu().numpy().reshape(nlay, ncol, 140)[:, c].T
            assert np.array_equal(got, ref[k][:, 0]), (k, c)
    for k in SUB:  # nothing past the arrays
        assert (buf[k][shift + n:] == -7.0).all() and (buf[k][:shift] == -7.0).all()
    assert torch.equal(d["reicmcl"], d["rei"]) and torch.equal(d["relqmcl"], d["rel"])


@pytest.mark.parametrize("ncol,nlay,icld,irng", [(5, 33, 3, 1), (4, 16, 3, 0), (3, 17, 2, 1), (9, 15, 4, 1)])
def test_shortwave_sub_columns(ctx, ncol, nlay, icld, irng):
    ctx.sw_ini(1004.0)
    st = _state(ncol, nlay, 90 + ncol)
    band = _sw_band(st, seed=icld)
    ref = pyoracle.mcica_subcol_sw(st, band, icld, 17, irng)
    got = ctx.mcica_subcol_sw(st, band, icld, 17, irng)
    for k in ref:
        assert np.array_equal(got[k], ref[k]), k
