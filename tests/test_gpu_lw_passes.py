"""Longwave batches through taumol's planes: column counts around the 32-column
tiles and the two columns of a unit, ragged grids in one batch, shallow and
deep columns, a batch that takes several passes over the planes, and the
network's rows at any address."""
import numpy as np
import pytest

import pyoracle
from brams_gb300 import rrtmg_lw as R
from brams_gb300 import surrogate as S
from brams_gb300.profiles import ProfileSpec, make_state

pytestmark = pytest.mark.gpu

FLUX_TOL, HR_TOL = 0.05, 0.01  # the solver's parity tolerances (W m-2, K/day)
OUTS = ("uflx", "dflx", "hr", "uflxc", "dflxc", "hrc", "duflx_dt", "duflxc_dt")


@pytest.fixture
def own():
    c = R.Context()
    yield c
    c.close()


def _solve(ctx, grids, seeds):
    import torch

    ctx.rrtmg_lw_batch_device([g.desc(seed0=s) for g, s in zip(grids, seeds)])
    torch.cuda.synchronize()
    assert ctx.sync_status() == 0
    return [g.outputs() for g in grids]


@pytest.mark.parametrize("shapes", [[(1, 3)], [(31, 45)], [(32, 38)], [(33, 60)], [(65, 7), (1, 128), (30, 46)],
                                    [(153, 38)], [(160, 46), (3, 45), (200, 5)], [(155, 230)]])
def test_ragged_batches_against_oracle(ctx, shapes):
    grids, refs, seeds = [], [], []
    for i, (ncol, nlay) in enumerate(shapes):
        st = make_state(ProfileSpec(ncol=ncol, nlay=nlay, seed=300 + i, t_noise=4.0, h2o_sigma=0.5))
        tauc = pyoracle.cldprop_columns(st)
        seeds.append(50 + 1000 * i)
        grids.append(S.DeviceGrid(st, tauc))
        refs.append(pyoracle.rrtmg_lw(st, pyoracle.mcica_per_column(st, tauc, icld=3, base_seed=seeds[-1]), icld=3))
    for got, ref in zip(_solve(ctx, grids, seeds), refs):
        for k in ("uflx", "dflx", "uflxc", "dflxc"):
            assert np.abs(got[k] - ref[k]).max() <= FLUX_TOL, k
        for k in ("hr", "hrc"):
            assert np.abs(got[k] - ref[k]).max() <= HR_TOL, k


def test_several_passes_equal_separate_calls(ctx):
    """More columns than the planes hold at once (their buffer is 1.5 GiB: about
    30,000 columns of 38 layers), in two grids: every column has the bits of a
    call of its own slice."""
    import torch

    from brams_gb300.shard import slice_grid

    n = [40001, 30003]
    grids = []
    for i, ncol in enumerate(n):
        g = S.DeviceGrid(make_state(ProfileSpec(ncol=1000, nlay=38, seed=7 + i, t_noise=4.0)))
        rep = (ncol + 999) // 1000
        for k, v in list(g.d.items()):
            g.d[k] = torch.cat([v] * rep, dim=-1)[..., :ncol].contiguous()
        g.d["tauc"] = torch.zeros((38, ncol, 16), dtype=torch.float64, device="cuda")
        g.ncol = ncol
        grids.append(g)
    whole = _solve(ctx, grids, [11, 99])
    for g, seed, ref in zip(grids, (11, 99), whole):
        for k in OUTS:
            g.d[k].zero_()
        d = g.desc(seed0=seed)
        for c0 in range(0, g.ncol, 9973):
            ctx.rrtmg_lw_batch_device([slice_grid(d, c0, min(c0 + 9973, g.ncol))])
        torch.cuda.synchronize()
        got = g.outputs()
        for k in OUTS:
            assert np.array_equal(got[k], ref[k]), k
    assert ctx.sync_status() == 0


@pytest.mark.parametrize("ncol", [7, 401])
def test_network_rows_on_any_address(ctx, ncol):
    """The learned batch reads its fp16 rows wherever they start: the same bits
    from rows on 4-byte boundaries and from rows one half word on."""
    import torch

    mlp = S.load(ctx)
    st = make_state(ProfileSpec(ncol=ncol, nlay=45, seed=5, t_noise=4.0))
    g = S.DeviceGrid(st, pyoracle.cldprop_columns(st))
    n = ncol * 45 * 140
    rows = torch.zeros((2, n + 4), dtype=torch.float16, device="cuda")
    flag = torch.zeros(ncol * 45, dtype=torch.uint8, device="cuda")
    mlp.infer(g.desc(), rows[0], rows[1], flag)
    got = []
    for shift in (0, 1):
        r = torch.zeros((2, n + 4), dtype=torch.float16, device="cuda")
        r[:, shift:shift + n] = rows[:, :n]
        ctx.rrtmg_lw_batch_device([g.desc(seed0=3, sur_tau=r[0, shift:], sur_frac=r[1, shift:], sur_flag=flag)])
        torch.cuda.synchronize()
        got.append(g.outputs())
    assert ctx.sync_status() == 0
    for k in OUTS:
        assert np.array_equal(got[0][k], got[1][k]), k
    mlp.close()


@pytest.mark.parametrize("nlay,variant,blocks,ok", [(45, 0, 6, True), (60, 0, 6, True), (60, 1, 7, True), (38, 3, 4, True),
                                                    (45, 0, 8, False), (45, 0, 0, False), (60, 3, 5, False)])
def test_shapes_pinned_in_column_blocks(ctx, nlay, variant, blocks, ok):
    """Shapes saved when a block was one column are taken, and run with as many units as fit."""
    saved = ctx.tuning(nlay, kind=R.KIND_FUSED)
    try:
        if not ok:
            with pytest.raises(R.RrtmgLwError):
                ctx.set_tuning(nlay, variant, blocks, kind=R.KIND_FUSED)
            return
        ctx.set_tuning(nlay, variant, blocks, kind=R.KIND_FUSED)
        got = ctx.tuning(nlay, kind=R.KIND_FUSED)
        assert got["variant"] == variant and 1 <= got["blocks_per_sm"] <= blocks
    finally:
        ctx.set_tuning(nlay, saved["variant"], saved["blocks_per_sm"], kind=R.KIND_FUSED)


# the largest nlay at which 7, 6, .. 1 blocks per SM have been taken since shapes can be kept
TAKEN = {7: 62, 6: 73, 5: 88, 4: 112, 3: 150, 2: 227, 1: 256}


@pytest.mark.parametrize("kind", [R.KIND_FUSED, R.KIND_FUSED | R.KIND_LEARNED])
@pytest.mark.parametrize("variant,most", [(0, 6), (1, 7), (2, 5), (3, 4)])
def test_which_shapes_are_taken(own, variant, most, kind):
    def taken(nlay, blocks):
        try:
            own.set_tuning(nlay, variant, blocks, kind=kind)
        except R.RrtmgLwError:
            return False
        return own.tuning(nlay, kind=kind)["blocks_per_sm"] <= blocks

    for blocks, nlay in TAKEN.items():
        for n in (nlay, nlay + 1):
            if n <= 256:
                assert taken(n, blocks) == (blocks <= most and n <= nlay), (blocks, n)
    assert not taken(38, 0) and not taken(38, most + 1)


def test_small_calls_equal_their_columns_in_a_large_one(ctx):
    """taumol's two register allocations (few blocks, many) give a column the same bits."""
    import torch

    from brams_gb300.shard import slice_grid

    st = make_state(ProfileSpec(ncol=1000, nlay=38, seed=17, t_noise=4.0, h2o_sigma=0.5))
    g = S.DeviceGrid(st, pyoracle.cldprop_columns(st))
    whole = _solve(ctx, [g], [5])[0]
    for k in OUTS:
        g.d[k].zero_()
    d = g.desc(seed0=5)
    for c0 in range(0, 1000, 40):
        ctx.rrtmg_lw_batch_device([slice_grid(d, c0, c0 + 40)])
    torch.cuda.synchronize()
    got = g.outputs()
    for k in OUTS:
        assert np.array_equal(got[k], whole[k]), k


@pytest.mark.parametrize("ncol,nlay", [(5, 96), (340, 97), (5, 207), (3, 256)])
def test_deep_columns_off_the_network(own, ncol, nlay):
    """Columns whose layers are all off the network have the plain path's bits, with
    one and several columns per hand-over block."""
    import torch

    g = S.DeviceGrid(make_state(ProfileSpec(ncol=ncol, nlay=nlay, seed=5, t_noise=4.0)))
    g.d["tauc"] = torch.full((nlay, ncol, 16), 3.0, dtype=torch.float64, device="cuda")
    g.d["tlay"] += 200.0
    ref = _solve(own, [g], [11])[0]
    for k in OUTS:
        g.d[k].zero_()
    net = S.load(own)
    net.batch([g.desc(seed0=11)])
    torch.cuda.synchronize()
    got = g.outputs()
    for k in OUTS:
        assert np.array_equal(got[k], ref[k]), k
    net.close()


@pytest.mark.parametrize("icld", [1, 2])
@pytest.mark.parametrize("nlay", [208, 229, 230])
def test_deep_band_clouds(own, nlay, icld):
    """Two columns a unit up to 229 layers, one above: the first columns of a call of
    155 against the oracle, and with the bits of a call of their own (a column a unit)."""
    st = make_state(ProfileSpec(ncol=155, nlay=nlay, seed=17, t_noise=3.0, cloud_prob=0.6))
    got = own.rrtmg_lw_nomcica(st, icld=icld)
    few = {k: np.asfortranarray(v[:4]) if getattr(v, "shape", (0,))[:1] == (155,) else v for k, v in st.items()}
    one = own.rrtmg_lw_nomcica(few, icld=icld)
    ref = pyoracle.rrtmg_lw_nomcica(few, icld=icld)
    for k in OUTS:
        assert np.array_equal(got[k][:4], one[k]), k
        tol = HR_TOL if k.startswith("hr") else 1e-3 if k.startswith("du") else FLUX_TOL
        assert np.abs(one[k] - ref[k]).max() <= tol, k
