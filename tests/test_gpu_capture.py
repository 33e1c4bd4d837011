"""Calls captured in a caller's own CUDA graph: the graph replays to the bits of
the direct call also after the context has served larger calls, and a call
captured with the scratch of a much smaller one makes more passes over it."""
import ctypes as C

import numpy as np
import pytest

import pyoracle
from brams_gb300 import rrtmg_lw as R
from brams_gb300 import surrogate as S
from brams_gb300.profiles import ProfileSpec, make_state
from test_sw import sw_mcica, sw_state

pytestmark = pytest.mark.gpu

NLAY = 38


def _tile(v, n, axis=-1):
    """The columns of a device array repeated up to n."""
    import torch

    m = v.shape[axis]
    return v.index_select(axis % v.dim(), torch.arange(n, device=v.device) % m).contiguous()


class Dropin:
    outs = R.OUT_ORDER

    def __init__(self, ctx, n, dt=0.0):
        st = make_state(ProfileSpec(ncol=131, nlay=NLAY, seed=4, t_noise=4.0, cloud_prob=0.6))
        st["tlay"] = st["tlay"] + dt
        mc = pyoracle.mcica_per_column(st, pyoracle.cldprop_columns(st), icld=3, base_seed=3)
        g = S.DeviceGrid(st)
        self.ctx, self.n, self.d = ctx, n, {k: _tile(v, n) for k, v in g.d.items()}
        for k in ("cldfmcl", "ciwpmcl", "clwpmcl", "taucmcl"):
            self.d[k] = _tile(S.dev(mc[k]), n, 1)
        self.d["reicmcl"], self.d["relqmcl"] = self.d["rei"], self.d["rel"]

    def run(self, stream):
        self.ctx.rrtmg_lw_device(self.n, NLAY, self.d, stream=stream)


class Nomcica(Dropin):
    def __init__(self, ctx, n, dt=0.0):
        import torch

        super().__init__(ctx, n, dt)
        self.d["tauc_band"] = torch.zeros((NLAY, n, 16), dtype=torch.float64, device="cuda")

    def run(self, stream):
        self.ctx.rrtmg_lw_nomcica_device(self.n, NLAY, self.d, stream=stream, icld=2)


class Batch(Dropin):
    def __init__(self, ctx, n, dt=0.0):
        import torch

        super().__init__(ctx, n, dt)
        self.d["tauc"] = torch.zeros((NLAY, n, 16), dtype=torch.float64, device="cuda")
        self.desc = R.grid_desc(n, NLAY, self.d, icld=3, cloud_mode=R.CLOUD_FUSED, seed0=9)

    def run(self, stream):
        self.ctx.rrtmg_lw_batch_device([self.desc], stream=stream)


class Learned(Batch):
    def __init__(self, ctx, n, dt=0.0):
        super().__init__(ctx, n, dt)
        self.d["tlay"][10, 7:90] += 200.0  # these columns are handed over
        if not hasattr(ctx, "net"):
            ctx.net = S.load(ctx)

    def run(self, stream):
        self.ctx.net.batch([self.desc], stream=stream)


class Shortwave:
    outs = R.SW_OUT
    bits = 32

    def __init__(self, ctx, n, dt=0.0):
        import torch

        st = sw_state(ncol=131, nlay=NLAY, seed=8, cloud_prob=0.6)
        st["tlay"] = st["tlay"] + dt
        mc = sw_mcica(st, seed=2)
        if not hasattr(ctx, "sw"):
            ctx.sw_ini(1004.0)
            ctx.sw = True
        ctx.sw_set_precision(self.bits)
        self.ctx, self.n = ctx, n
        self.d = {k: _tile(S.dev(st[k]), n) for k in (*R.SW_STATE, "tauaer_sw", "ssaaer_sw", "asmaer_sw")}
        self.d.update({k: _tile(S.dev(mc[k]), n, 1 if mc[k].ndim == 3 else -1) for k in R.SW_CLOUD})
        for k in R.SW_OUT:
            self.d[k] = torch.zeros((NLAY + 1 if "flx" in k else NLAY, n), dtype=torch.float64, device="cuda")

    def run(self, stream):
        p = lambda k: self.d[k].data_ptr()
        ic, ia = C.c_int(3), C.c_int(10)
        rc = self.ctx.L.gb_rrtmg_sw_device(
            self.ctx.h, C.c_void_p(stream or 0), self.n, NLAY, C.byref(ic), C.byref(ia), *[p(k) for k in R.SW_STATE],
            1.0, 0, 1368.22, -1, 2, 3, 1, *[p(k) for k in R.SW_CLOUD],
            *[p(k) for k in ("tauaer_sw", "ssaaer_sw", "asmaer_sw")], None, *[p(k) for k in R.SW_OUT], self.n, self.n, None)
        assert rc == 0


class Shortwave64(Shortwave):
    bits = 64


def _results(c):
    import torch

    torch.cuda.synchronize()
    return {k: c.d[k].cpu().numpy().copy() for k in c.outs}


def _direct(c):
    c.run(None)
    return _results(c)


def _capture(c):
    import torch

    torch.cuda.synchronize()
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        c.run(s.cuda_stream)
    return g


def _replay(g, c):
    for k in c.outs:
        c.d[k].zero_()
    g.replay()
    return _results(c)


def _same(a, b):
    for k in b:
        assert np.array_equal(a[k], b[k]), k


@pytest.fixture
def own():
    c = R.Context()
    yield c
    if hasattr(c, "net"):
        c.net.close()
    c.close()


@pytest.mark.parametrize("kind", [Dropin, Nomcica, Batch, Learned, Shortwave, Shortwave64])
def test_a_graph_outlives_larger_calls(own, kind):
    small, mid, large = kind(own, 300), kind(own, 1300, 1.0), kind(own, 5000, 2.0)
    ref = {c: _direct(c) for c in (small,)}
    g = _capture(small)
    _same(_replay(g, small), ref[small])
    ref[mid] = _direct(mid)
    g2 = _capture(mid)
    ref[large] = _direct(large)
    for _ in range(2):
        _same(_replay(g, small), ref[small])
        _same(_replay(g2, mid), ref[mid])
        _same(_direct(large), ref[large])
    assert own.sync_status() == 0


@pytest.mark.parametrize("kind", [Dropin, Shortwave, Shortwave64])
def test_capture_with_the_scratch_of_a_smaller_call(own, kind):
    """33 columns leave the least scratch a call runs with: 2,101 columns take it in ten passes and more."""
    fresh = R.Context()
    ref = _direct(kind(fresh, 2101))
    _direct(kind(own, 33, 1.0))
    c = kind(own, 2101)
    g = _capture(c)
    _same(_replay(g, c), ref)
    _same(_direct(c), ref)
    assert own.sync_status() == 0
    fresh.close()
