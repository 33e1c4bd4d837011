"""The work that users of this framework have it do, as timed cases.

Every case goes through the public Python entry points of brams_gb300 on
device arrays in the reference's Fortran layouts (a (ncol, nlay) array is held
as a torch tensor of shape (nlay, ncol)).  Inputs follow the generator of
brams_gb300/profiles.py (same distributions), drawn on the device from the
seed; clouds, temperatures and humidities differ from column to column,
pressures are those of the generator's levels.  The host-array call rrtmg_lw is
the drop-in case plus copies of pageable memory, whose time varies several-fold
from pass to pass on the same inputs, so it is not among the cases.

Kinds of case ("do"):

* ``batch``    -- rrtmg_lw_batch_device: plain gas optics, McICA clouds made in
                  the kernel, one or several grids per call;
* ``learned``  -- Mlp.batch: the same call on the learned gas optics;
* ``dropin``   -- rrtmg_lw_device on the reference's McICA arrays;
* ``nomcica``  -- rrtmg_lw_nomcica_device (band clouds, cldprop included);
* ``subcol``   -- mcica_subcol_lw_device, the sub-column generator;
* ``sw``       -- rrtmg_sw_device in fp32 or fp64;
* ``brams``    -- the whole caller-side chain: pack, cldprop, rrtmg_lw batch,
                  write-back of the theta tendency and surface flux;
* ``train``    -- forward and backward of the gas-optics network on a batch.

exact() gives the sub-columns and the network's loss and gradients in 64 bits.
The solvers have no 64-bit value here: it would be a second statement of
sixteen gas-optics bands and two radiative transfers (some thousands of lines),
and their outputs are 64-bit arrays, which are compared as such.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from brams_gb300 import rrtmg_lw as R
from brams_gb300 import surrogate as S
from brams_gb300.profiles import CCL4, CFC11, CFC12, CFC22, O2_VMR, base_profile

LEVEL_OUT = ("uflx", "dflx", "uflxc", "dflxc", "duflx_dt", "duflxc_dt")
SUBCOL_LW = ("cldfmcl", "ciwpmcl", "clwpmcl", "taucmcl")
SUBCOL_SW = ("cldfmcl", "ciwpmcl", "clwpmcl", "taucmcl", "ssacmcl", "asmcmcl", "fsfcmcl")
NG_LW = (10, 12, 16, 14, 16, 8, 12, 8, 12, 6, 8, 8, 4, 2, 2, 2)  # g-points per longwave band

_kept = {}  # the context and the networks a program opens once


def _ctx():
    if "ctx" not in _kept:
        _kept["ctx"] = R.Context()
        _kept["ctx"].sw_ini(1004.0)
    return _kept["ctx"]


def _network():
    if "mlp" not in _kept:
        _kept["mlp"] = S.load(_ctx())
    return _kept["mlp"]


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest calls: one MPI rank's sub-domain of a small grid, where latency and launches count
        {"name": "batch 8x8x38", "do": "batch", "grids": "64x38"},
        # ragged nested grids of one model step in one call (benchmark: 200x180, 150x150 and 97x97 columns)
        {"name": "batch nested", "do": "batch", "grids": "36000x45,22500x45,9409x38"},
        # a chunk of the 2048x1024x60 ensemble workload, plain gas optics
        {"name": "batch 131072x60", "do": "batch", "grids": "131072x60"},
        # the headline: the same on the learned gas optics, four members per call
        {"name": "learned 4x32768x60", "do": "learned", "grids": "32768x60,32768x60,32768x60,32768x60"},
        # the drop-in call on the reference's McICA arrays at the largest stated grid (360x300x45)
        {"name": "dropin 360x300x45", "do": "dropin", "ncol": 108000, "nlay": 45},
        # ... and at the oracle configuration (64x64x38), an ordinary sub-domain
        {"name": "dropin 64x64x38", "do": "dropin", "ncol": 4096, "nlay": 38},
        # the non-McICA build of the driver, maximum/random overlap
        {"name": "nomcica 150x150x45", "do": "nomcica", "ncol": 22500, "nlay": 45, "icld": 2},
        # the sub-column generator that feeds the drop-in call
        {"name": "subcol 200x180x45", "do": "subcol", "ncol": 36000, "nlay": 45, "icld": 3},
        # the shortwave solver BRAMS calls right after, in its default precision ...
        {"name": "sw fp32 200x180x45", "do": "sw", "ncol": 36000, "nlay": 45, "bits": 32},
        # ... and in fp64 throughout
        {"name": "sw fp64 64x64x45", "do": "sw", "ncol": 4096, "nlay": 45, "bits": 64},
        # one radiation step of the model: fields in, theta tendency and surface flux out
        {"name": "brams 97x97x38", "do": "brams", "mxp": 99, "myp": 99, "mzp": 39},
        # one batch of training the learned gas optics (forward and backward)
        {"name": "train 16384", "do": "train", "rows": 16384},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    do = rng.choice(["batch", "batch", "learned", "dropin", "dropin", "nomcica", "subcol", "sw", "sw", "brams", "train"])
    nlay = rng.randint(38, 60)
    if do in ("batch", "learned"):
        n = rng.choice([1, 1, 2, 3, 4])
        left, grids = 131072 * 60, []
        for _ in range(n):
            nlay = rng.randint(38, 60)
            top = left // (n * nlay)
            grids.append("%dx%d" % (_log_int(rng, 16, top), nlay))
        return {"do": do, "grids": ",".join(grids)}
    if do == "dropin":
        return {"do": do, "ncol": _log_int(rng, 16, 108000 * 45 // nlay), "nlay": nlay}
    if do == "nomcica":
        return {"do": do, "ncol": _log_int(rng, 16, 22500 * 45 // nlay), "nlay": nlay, "icld": rng.choice([1, 2])}
    if do == "subcol":
        icld = rng.choice([1, 2, 3])
        return {"do": do, "ncol": _log_int(rng, 16, (36000 if icld == 3 else 4000) * 45 // nlay), "nlay": nlay,
                "icld": icld}
    if do == "sw":
        bits = rng.choice([32, 64])
        return {"do": do, "ncol": _log_int(rng, 16, (36000 if bits == 32 else 4096) * 45 // nlay), "nlay": nlay,
                "bits": bits}
    if do == "brams":
        return {"do": do, "mxp": rng.randint(5, 99), "myp": rng.randint(5, 99), "mzp": rng.randint(31, 39)}
    return {"do": do, "rows": 8 * _log_int(rng, 128, 2048)}


def _grids(case):
    return [tuple(int(v) for v in g.split("x")) for g in case["grids"].split(",")]


# ------------------------------------------------------------------ inputs
class _Draw:
    """Seeded values on the device, in memory order (nlay, ncol)."""

    def __init__(self, seed, salt=0):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed * 1000 + salt)

    def u(self, *shape, lo=0.0, hi=1.0, dtype=torch.float64):
        return lo + (hi - lo) * torch.rand(shape, generator=self.g, device="cuda", dtype=dtype)

    def n(self, *shape, dtype=torch.float64):
        return torch.randn(shape, generator=self.g, device="cuda", dtype=dtype)


def _columns(ncol, nlay, seed, salt=0):
    """Column state and layer clouds (profiles.make_state's distributions)."""
    r = _Draw(seed, salt)
    ptop = 5.0 if nlay >= 60 else 10.0
    plev, play, tlev, tlay, _, zmid = base_profile(nlay, ptop)
    col = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()[:, None].expand(len(a), ncol).contiguous()
    const = lambda v: torch.full((nlay, ncol), v, dtype=torch.float64, device="cuda")
    d = {"plev": col(plev), "play": col(play), "tlev": col(tlev)}
    d["tlay"] = col(tlay) + 4.0 * r.n(nlay, ncol)
    d["tsfc"] = float(tlev[0]) + r.n(ncol)
    d["h2ovmr"] = (col(0.015 * np.exp(-zmid / 2.5)) * torch.exp(0.5 * r.n(nlay, ncol))).clamp_(3.0e-6, 0.05)
    d["o3vmr"] = col(8.0e-6 * np.exp(-0.5 * ((zmid - 25.0) / 6.0) ** 2) + 2.0e-8)
    for k, v in (("co2vmr", 400.0e-6), ("ch4vmr", 1.8e-6), ("n2ovmr", 0.32e-6), ("o2vmr", O2_VMR),
                 ("cfc11vmr", CFC11), ("cfc12vmr", CFC12), ("cfc22vmr", CFC22), ("ccl4vmr", CCL4)):
        d[k] = const(v)
    d["emis"] = r.u(16, ncol, lo=0.95, hi=1.0)
    d["tauaer"] = torch.zeros((16, nlay, ncol), dtype=torch.float64, device="cuda")
    lay = torch.arange(1, nlay + 1, device="cuda")[:, None]
    present = (r.u(nlay, ncol) < 0.3) & (lay >= 5) & (lay <= 20)
    zero = torch.zeros((), dtype=torch.float64, device="cuda")
    path = torch.exp(math.log(50.0) - 0.32 + 0.8 * r.n(nlay, ncol))
    cold = d["tlay"] < 253.0
    d["cldfrac"] = torch.where(present, r.u(nlay, ncol), zero)
    d["ciwp"] = torch.where(present & cold, path, zero)
    d["clwp"] = torch.where(present & ~cold, path, zero)
    d["rei"], d["rel"] = const(50.0), const(10.0)
    return d


def _lw_out(d, nlay, ncol):
    for k in LEVEL_OUT:
        d[k] = torch.zeros((nlay + 1, ncol), dtype=torch.float64, device="cuda")
    for k in ("hr", "hrc"):
        d[k] = torch.zeros((nlay, ncol), dtype=torch.float64, device="cuda")


def _band_depth(d, nlay, ncol):
    """cldprop's cloud optical depth per band, which the generator and the fused batch take."""
    d["tauc"] = torch.zeros((nlay, ncol, 16), dtype=torch.float64, device="cuda")
    _ctx().cldprop_lw_device(ncol, nlay, {**{k: d[k] for k in ("cldfrac", "ciwp", "clwp", "rei", "rel")},
                                          "taucloud": d["tauc"]})


def _subcol_arrays(d, nlay, ncol):
    for k in SUBCOL_LW:
        d[k] = torch.empty((nlay, ncol, 140), dtype=torch.float64, device="cuda")
    for k in ("reicmcl", "relqmcl"):
        d[k] = torch.empty((nlay, ncol), dtype=torch.float64, device="cuda")


def _subcolumns(d, nlay, ncol, seed):
    _band_depth(d, nlay, ncol)
    _subcol_arrays(d, nlay, ncol)
    _ctx().mcica_subcol_lw_device(ncol, nlay, d, icld=3, permuteseed=seed)


def _sw_state(ncol, nlay, seed):
    d = _columns(ncol, nlay, seed)
    r = _Draw(seed, 7)
    for k in ("asdir", "asdif", "aldir", "aldif"):
        d[k] = r.u(ncol, lo=0.05, hi=0.4)
    d["coszen"] = r.u(ncol, lo=0.05, hi=1.0)
    d["tauaer_sw"] = r.u(14, nlay, ncol, lo=0.0, hi=0.05)
    d["ssaaer_sw"] = r.u(14, nlay, ncol, lo=0.8, hi=0.99)
    d["asmaer_sw"] = r.u(14, nlay, ncol, lo=0.5, hi=0.8)
    b = {k: r.u(nlay, ncol, 14, lo=lo, hi=hi) for k, lo, hi in
         (("tauc", 0.5, 10.0), ("ssac", 0.9, 1.0), ("asmc", 0.7, 0.9), ("fsfc", 0.0, 0.5))}
    m = {k: torch.empty((nlay, ncol, 112), dtype=torch.float64, device="cuda") for k in SUBCOL_SW}
    m["reicmcl"] = torch.empty((nlay, ncol), dtype=torch.float64, device="cuda")
    m["relqmcl"] = torch.empty((nlay, ncol), dtype=torch.float64, device="cuda")
    ctx, ir = _ctx(), C.c_int(1)
    rc = ctx.L.gb_mcica_subcol_sw_device(
        ctx.h, None, ncol, nlay, 3, seed & 0xFFFFFF, C.byref(ir),
        *[d[k].data_ptr() for k in ("play", "cldfrac", "ciwp", "clwp", "rei", "rel")],
        *[b[k].data_ptr() for k in ("tauc", "ssac", "asmc", "fsfc")], None,
        *[m[k].data_ptr() for k in ("cldfmcl", "ciwpmcl", "clwpmcl", "reicmcl", "relqmcl", "taucmcl", "ssacmcl",
                                    "asmcmcl", "fsfcmcl")], ncol, 1)
    if rc:
        raise RuntimeError("mcica_subcol_sw: status %d" % rc)
    torch.cuda.synchronize()  # the band values go out of scope here
    o = {k: torch.zeros((nlay + 1 if "flx" in k else nlay, ncol), dtype=torch.float64, device="cuda")
         for k in R.SW_OUT}
    return d, m, o


def _brams_fields(mzp, mxp, myp, seed):
    """Model fields in BRAMS's default-real Fortran arrays: memory order (myp, mxp, mzp)."""
    cp, rgas, p00, sigma = 1004.0, 287.0, 1.0e5, 5.6696e-8
    r = _Draw(seed, 3)
    f3 = (myp, mxp, mzp)
    z = (torch.arange(mzp, device="cuda", dtype=torch.float64) - 0.5) * 400.0
    ps, ts = r.u(myp, mxp, lo=95000.0, hi=102000.0), r.u(myp, mxp, lo=280.0, hi=302.0)
    p = ps[..., None] * torch.exp(-z / 8000.0)
    t = (ts[..., None] - 6.5e-3 * z).clamp(min=212.0) + 0.5 * r.n(*f3)
    exner = cp * (p / p00) ** (rgas / cp)
    pp = 0.3 * r.n(*f3)
    rv = 0.012 * torch.exp(-z.clamp(min=0.0) / 2500.0) * torch.exp(0.2 * r.n(*f3))
    k = torch.arange(mzp, device="cuda")
    cloudy = (r.u(*f3) < 0.3) & (k >= 2) & (k < min(mzp - 1, 24))
    on = lambda cond, v: torch.where(cond, v, torch.zeros_like(v))
    f = {"pi0": exner - pp, "pp": pp, "theta": t * cp / exner, "rv": rv, "cldf": on(cloudy, r.u(*f3, lo=0.05)),
         "lwl": on(cloudy & (t > 253.0), 50.0 * torch.exp(0.8 * r.n(*f3))),
         "iwl": on(cloudy & (t < 263.0), 20.0 * torch.exp(0.8 * r.n(*f3))),
         "rel": r.u(*f3, lo=5.0, hi=20.0), "rei": r.u(*f3, lo=20.0, hi=120.0),
         "rlongup": sigma * ts ** 4, "albedt": r.u(myp, mxp, lo=0.02, hi=0.1)}
    return {key: v.to(torch.float32).contiguous() for key, v in f.items()}


def _batch_desc(d, ncol, nlay, seed0):
    arrays = dict(d)
    arrays["reicmcl"], arrays["relqmcl"] = d["rei"], d["rel"]
    return R.grid_desc(ncol, nlay, arrays, icld=3, cloud_mode=R.CLOUD_FUSED, seed0=seed0)


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    do = case["do"]
    seed0 = seed * 7919 + 11
    s = {"do": do, "ctx": _ctx()}
    if do in ("batch", "learned"):
        s["grids"], s["descs"] = [], []
        for i, (ncol, nlay) in enumerate(_grids(case)):
            d = _columns(ncol, nlay, seed, salt=10 + i)
            _band_depth(d, nlay, ncol)
            _lw_out(d, nlay, ncol)
            s["grids"].append(d)
            s["descs"].append(_batch_desc(d, ncol, nlay, seed0 + 1000003 * i))
        if do == "learned":
            s["mlp"] = _network()
    elif do == "train":
        r = _Draw(seed, 5)
        rows = case["rows"]
        x = torch.zeros((rows, 16), dtype=torch.float64, device="cuda")
        x[:, :9] = r.n(rows, 9)
        t = torch.zeros((rows, 288), dtype=torch.float32, device="cuda")
        t[:, :280] = r.n(rows, 280)
        s.update(mlp=_network(), rows=rows, x=x.to(torch.bfloat16), t=t,
                 grad=torch.zeros(R.MLP_NPARAM, dtype=torch.float32, device="cuda"),
                 loss=torch.zeros(1, dtype=torch.float32, device="cuda"))
    elif do == "brams":
        mzp, mxp, myp = case["mzp"], case["mxp"], case["myp"]
        box = (2, mxp - 1, 2, myp - 1)  # the interior of the sub-domain, as BRAMS passes it
        ncol, nlay = (mxp - 2) * (myp - 2), mzp - 1
        d = _brams_fields(mzp, mxp, myp, seed)
        rows = {"plev": nlay + 1, "tlev": nlay + 1, "tsfc": 1, "emis": 16}
        for k in R.Context.PACK_OUT:
            d[k] = torch.zeros((rows.get(k, nlay), ncol), dtype=torch.float64, device="cuda")
        p = 1000.0 * np.exp(-(np.arange(nlay) * 400.0) / 8000.0)  # ozone from a profile on the model's levels
        o3 = 8.0e-6 * np.exp(-np.log(p / 30.0) ** 2 / 2.0) + 2.0e-8
        d["o3vmr"] = torch.from_numpy(o3).cuda()[:, None].expand(nlay, ncol).contiguous()
        d["tauaer"] = torch.zeros((16, nlay, ncol), dtype=torch.float64, device="cuda")
        d["tauc"] = torch.zeros((nlay, ncol, 16), dtype=torch.float64, device="cuda")
        _lw_out(d, nlay, ncol)
        arrays = dict(d)
        arrays["reicmcl"], arrays["relqmcl"] = d["reic"], d["relq"]
        s.update(d=d, dims=(mzp, mxp, myp), box=box, ncol=ncol, nlay=nlay,
                 desc=R.grid_desc(ncol, nlay, arrays, icld=3, cloud_mode=R.CLOUD_FUSED, seed0=seed0),
                 fthrd=torch.zeros((myp, mxp, mzp), dtype=torch.float32, device="cuda"),
                 rlong=torch.zeros((myp, mxp), dtype=torch.float32, device="cuda"))
    else:
        ncol, nlay = case["ncol"], case["nlay"]
        s.update(ncol=ncol, nlay=nlay)
        if do == "sw":
            s["d"], s["m"], s["o"] = _sw_state(ncol, nlay, seed)
            s["bits"] = case["bits"]
        else:
            s["d"] = d = _columns(ncol, nlay, seed)
            s["seed0"] = seed0 & 0xFFFFFF
            if do == "dropin":
                _subcolumns(d, nlay, ncol, s["seed0"])
                _lw_out(d, nlay, ncol)
            elif do == "nomcica":
                d["tauc_band"] = torch.zeros((nlay, ncol, 16), dtype=torch.float64, device="cuda")
                _lw_out(d, nlay, ncol)
                s["icld"] = case["icld"]
            else:  # subcol
                _band_depth(d, nlay, ncol)
                _subcol_arrays(d, nlay, ncol)
                s["icld"] = case["icld"]
    return s


def run(s):
    ctx, do = s["ctx"], s["do"]
    if do == "batch":
        ctx.rrtmg_lw_batch_device(s["descs"])
        return [{k: d[k] for k in R.OUT_ORDER} for d in s["grids"]]
    if do == "learned":
        s["mlp"].batch(s["descs"])
        return [{k: d[k] for k in R.OUT_ORDER} for d in s["grids"]]
    if do == "train":
        s["mlp"].gradients(s["rows"], s["x"], s["t"], s["grad"], s["loss"])
        return {"grad": s["grad"], "loss": s["loss"]}
    if do == "brams":
        d, ncol, nlay, dims, box = s["d"], s["ncol"], s["nlay"], s["dims"], s["box"]
        ctx.rtm_pack_lw_device(*dims, box, d)
        ctx.cldprop_lw_device(ncol, nlay, {"cldfrac": d["cldfrac"], "ciwp": d["ciwp"], "clwp": d["clwp"],
                                           "rei": d["reic"], "rel": d["relq"], "taucloud": d["tauc"]})
        ctx.rrtmg_lw_batch_device([s["desc"]])
        ctx.rtm_unpack_lw_device(*dims, box, d["hr"], d["dflx"], s["fthrd"], s["rlong"])
        return {"fthrd": s["fthrd"], "rlong": s["rlong"], **{k: d[k] for k in R.OUT_ORDER}}
    ncol, nlay, d = s["ncol"], s["nlay"], s["d"]
    if do == "dropin":
        ctx.rrtmg_lw_device(ncol, nlay, d)
        return {k: d[k] for k in R.OUT_ORDER}
    if do == "nomcica":
        ctx.rrtmg_lw_nomcica_device(ncol, nlay, d, icld=s["icld"])
        return {k: d[k] for k in R.OUT_ORDER}
    if do == "subcol":
        ctx.mcica_subcol_lw_device(ncol, nlay, d, icld=s["icld"], permuteseed=s["seed0"])
        return {k: d[k] for k in SUBCOL_LW + ("reicmcl", "relqmcl")}
    # the shortwave solver: the C entry point, as a program with device arrays calls it
    m, o = s["m"], s["o"]
    ctx.sw_set_precision(s["bits"])
    ic, ia = C.c_int(3), C.c_int(10)
    rc = ctx.L.gb_rrtmg_sw_device(
        ctx.h, None, ncol, nlay, C.byref(ic), C.byref(ia), *[d[k].data_ptr() for k in R.SW_STATE], 1.0, 0, 1368.22,
        -1, 2, 3, 1, *[m[k].data_ptr() for k in R.SW_CLOUD],
        *[d[k].data_ptr() for k in ("tauaer_sw", "ssaaer_sw", "asmaer_sw")], None,
        *[o[k].data_ptr() for k in R.SW_OUT], ncol, ncol, None)
    if rc:
        raise RuntimeError("rrtmg_sw: status %d" % rc)
    return {k: o[k] for k in R.SW_OUT}


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    """Bytes: every input read once and every output written once.  FLOPs: the
    operations of the FP64 restatement per column (565e3 at 60 layers, in
    proportion to the layers; shortwave 1.40e6 at 45), the network's matrix
    products, the generator's compares."""
    do = case["do"]
    if do in ("batch", "learned"):
        b = f = 0.0
        for ncol, nlay in _grids(case):
            b += ncol * 8.0 * (13 * nlay + 2 * (nlay + 1) + 1 + 16 + 32 * nlay + 5 * nlay + 6 * (nlay + 1) + 2 * nlay)
            f += ncol * nlay * (567e3 / 60 if do == "batch" else 331e3 / 60 + 2 * 139520.0)
        return {"bytes": b, "flops": f}
    if do == "train":
        rows = case["rows"]
        return {"bytes": rows * (32.0 + 4 * 288) + 4.0 * R.MLP_NPARAM * 2, "flops": 6.0 * rows * (16 + 128 + 128 + 288) * 128}
    if do == "brams":
        ncol, nlay = (case["mxp"] - 2) * (case["myp"] - 2), case["mzp"] - 1
        state = 8.0 * (21 * nlay + 2 * (nlay + 1) + 17 + 32 * nlay)
        return {"bytes": ncol * (4.0 * (9 * nlay + 2) + 2 * state + 8.0 * (8 * nlay + 6) + 4 * nlay + 4),
                "flops": ncol * nlay * 567e3 / 60}
    ncol, nlay = case["ncol"], case["nlay"]
    if do == "dropin":
        return {"bytes": ncol * 8.0 * (600 * nlay + 25), "flops": ncol * nlay * 567e3 / 60}
    if do == "nomcica":
        return {"bytes": ncol * 8.0 * (35 * nlay + 2 * (nlay + 1) + 17 + 16 * nlay + 8 * nlay + 6),
                "flops": ncol * nlay * 567e3 / 60}
    if do == "subcol":
        return {"bytes": ncol * nlay * 8.0 * (4 * 140 + 2 + 6 + 16), "flops": ncol * nlay * 140.0}
    return {"bytes": ncol * 8.0 * (6 * 112 * nlay + 2 * nlay + 42 * nlay + 12 * nlay + 6 + 6 * nlay),
            "flops": ncol * nlay * 1.40e6 / 45}


# ------------------------------------------------------------------ 64-bit values
def exact(case, seed):
    if case["do"] == "subcol":
        return _exact_subcol(case, seed)
    if case["do"] == "train":
        return _exact_train(case, seed)
    return None


def _exact_subcol(case, seed):
    """mcica_subcol_lw with one Mersenne-twister sequence per column (seed + column)."""
    s = prepare(case, seed)
    d, ncol, nlay, icld = s["d"], case["ncol"], case["nlay"], case["icld"]
    per = 1 if icld == 3 else nlay
    bits = np.empty((ncol, 140 * per), dtype=np.uint32)
    for c in range(ncol):
        bits[c] = np.random.RandomState(s["seed0"] + c).randint(0, 1 << 32, 140 * per, dtype=np.uint32)
    x = torch.from_numpy(bits.astype(np.float64) / 4294967295.0).cuda()
    x = (x[:, :, None].expand(ncol, 140, nlay) if icld == 3 else x.reshape(ncol, 140, nlay)).permute(2, 0, 1)
    frac = torch.where(d["cldfrac"] < 1.0e-20, torch.zeros_like(d["cldfrac"]), d["cldfrac"])
    if icld == 2:  # maximum-random: the draw of the layer below is kept where it was cloudy
        x = x.clone()
        for k in range(1, nlay):
            below = 1.0 - frac[k - 1][:, None]
            x[k] = torch.where(x[k - 1] > below, x[k - 1], x[k] * below)
    on = (x >= (1.0 - frac)[:, :, None]).to(torch.float64)
    band = torch.tensor([b for b, n in enumerate(NG_LW) for _ in range(n)], device="cuda")
    return {"cldfmcl": on, "ciwpmcl": on * d["ciwp"][:, :, None], "clwpmcl": on * d["clwp"][:, :, None],
            "taucmcl": on * d["tauc"][:, :, band], "reicmcl": d["rei"], "relqmcl": d["rel"]}


def _exact_train(case, seed):
    """Mean square loss of the 280 outputs and its gradient, the network in 64 bits throughout."""
    s = prepare(case, seed)
    p = torch.from_numpy(s["mlp"].params()[0].astype(np.float64)).cuda().requires_grad_()
    shapes, at, w = [(16, 128), (128,), (128, 128), (128,), (128, 128), (128,), (128, 288), (288,)], 0, []
    for sh in shapes:
        n = int(np.prod(sh))
        w.append(p[at:at + n].reshape(sh))
        at += n
    a = s["x"].to(torch.float64)
    for k in range(3):
        a = torch.nn.functional.silu(a @ w[2 * k] + w[2 * k + 1])
    y = a @ w[6] + w[7]
    loss = ((y - s["t"].to(torch.float64))[:, :280] ** 2).sum() / (case["rows"] * 280.0)
    loss.backward()
    return {"grad": p.grad, "loss": loss.detach().reshape(1)}
