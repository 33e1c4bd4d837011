"""The kernels' own arithmetic against the operators and against fp64, element
by element (arith.cu)."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from brams_gb300 import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def arith(tmp_path_factory):
    src = os.path.join(os.path.dirname(os.path.abspath(__file__)), "arith.cu")
    so = str(tmp_path_factory.mktemp("arith") / "libarith.so")
    subprocess.run([build.nvcc(), *build.ARCH, "-O3", "-std=c++17", "--extended-lambda", "-shared", "-Xcompiler", "-fPIC",
                    "-o", so, src], check=True)
    L = C.CDLL(so)

    def call(name, *args):
        import torch

        a = [C.c_void_p(x.data_ptr()) if isinstance(x, torch.Tensor) else x for x in args]
        assert getattr(L, name)(*a) == 0, name

    return call


def _floats(n, lo, hi, seed):
    """Positive floats, uniform in the exponent, with random significands."""
    rng = np.random.default_rng(seed)
    return np.exp2(rng.uniform(lo, hi, n)).astype(np.float32)


def test_table_quotient_and_index(arith):
    """od / (bpade + od) within the 2 ulp of PTX's approximate division (counted,
    as CUDA states its errors, from the correctly rounded quotient), the index
    that of the exact quotient or its neighbour where that is within 3e-7 of a
    half; 0 for optical depths beyond 2^126."""
    import torch

    inf = np.float32(np.inf)
    od = np.concatenate([[0.0, 1e-45, 0.06, 3.597, 1e4, 3e38, inf], _floats(1 << 20, -126, 128, 1),
                         _floats(1 << 20, -8, 12, 2)]).astype(np.float32)
    d = torch.from_numpy(od).cuda()
    q = torch.empty_like(d)
    itr = torch.empty(d.numel(), dtype=torch.int32, device="cuda")
    arith("arith_tbl", d, q, itr, C.c_longlong(d.numel()))
    q, itr = q.cpu().numpy(), itr.cpu().numpy()
    with np.errstate(all="ignore"):
        b = np.float32(np.float32(1.0) / np.float32(0.278)) + od
        ref = od.astype(np.float64) / b.astype(np.float64)
    near = b <= np.float32(2.0 ** 126)
    far = (b > np.float32(2.0 ** 126)) & (od < inf)
    normal = near & (ref >= 2.0 ** -126)
    rounded = ref[normal].astype(np.float32)
    assert (np.abs(q[normal].astype(np.float64) - rounded) <= 2.0 * np.spacing(rounded).astype(np.float64)).all()
    assert (q[near & ~normal] <= 2.0 ** -126).all()
    assert (q[far] == 0.0).all() and np.isnan(q[od == inf]).all()
    assert (itr[far] == 0).all() and (itr[od == inf] == 0).all()
    x = 10000.0 * ref[near] + 0.5
    assert ((itr[near] <= x + 3e-3) & (itr[near] > x - 1.0 - 3e-3)).all()
    assert itr.min() >= 0 and itr.max() <= 10000


@pytest.mark.parametrize("eb", [0, -59, 59])
def test_fp32_division_rounds_as_the_operator(arith, eb):
    """div_mid.  By Markstein's theorem the corrected quotient is the rounded one
    where the reciprocal is, unless the divisor's significand is all ones: the
    divisors where either fails are taken with every dividend's significand, all
    divisors with some dividends."""
    import torch

    rng = np.random.default_rng(3)
    a = np.exp2(rng.uniform(-30.0, 30.0, 64)).astype(np.float32)
    bad = torch.zeros(2, dtype=torch.int32, device="cuda")
    exact = torch.zeros(1 << 23, dtype=torch.uint8, device="cuda")
    arith("arith_div_cols", torch.from_numpy(a).cuda(), eb, bad, exact, 64)
    off = torch.nonzero(exact == 0).flatten().cpu().numpy()
    assert bad[0].item() == 0, (bad[0].item(), hex(bad[1].item() & 0xFFFFFFFF))
    assert len(off) <= 256
    t = np.concatenate([off, [0x7FFFFF, 0x7FFFFE, 0, 1]]).astype(np.int32)
    arith("arith_div_rows", torch.from_numpy(t).cuda(), 0, eb, bad, C.c_longlong(len(t)))
    assert bad[0].item() == 0, (bad[0].item(), hex(bad[1].item() & 0xFFFFFFFF))


def test_fp32_division_over_exponents(arith):
    """Operands 2^-60 to 2^60 and the quotients they give, among them powers of two and 0 / b."""
    import torch

    n = 1 << 22
    a, b = _floats(n, -60, 60, 5), _floats(n, -60, 60, 6)
    a[:1000], b[500:2000], a[3000:3100] = 1.0, 2.0, 0.0
    a[4000:5000] = b[4000:5000]
    d = [torch.from_numpy(v).cuda() for v in (a, b)]
    q, ref = torch.empty_like(d[0]), torch.empty_like(d[0])
    arith("arith_div", *d, q, ref, C.c_longlong(n))
    assert torch.equal(q, ref)


def test_fp64_reciprocal_root_and_constant_division(arith):
    """rcp64 and sqrt64 within one unit of the correctly rounded operators for every
    exponent, and the operators' own results where the estimates do not reach
    (zeros, subnormals, infinities, negative roots); div_c the operator's bits."""
    import torch

    rng = np.random.default_rng(9)
    n = 1 << 21
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-1073, 1023, n)) * rng.choice([-1.0, 1.0], n, p=[0.2, 0.8])
    x[: n // 4] = rng.uniform(-400.0, 400.0, n // 4)  # temperature differences
    x[-8:] = [0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, 1.7e308, 2.0 ** -959]
    d = torch.from_numpy(x).cuda()
    out = [torch.empty((n, 2), dtype=torch.float64, device="cuda") for _ in range(5)]
    arith("arith_f64", d, *out, C.c_longlong(n))
    rcp, root, *divs = [o.cpu().numpy() for o in out]

    def units(v):
        same = (v[:, 0] == v[:, 1]) | (np.isnan(v[:, 0]) & np.isnan(v[:, 1]))
        diff = np.abs(v[:, 0].view(np.int64) - v[:, 1].view(np.int64))
        return np.where(same, 0, diff)

    reach = (np.abs(x) >= 2.0 ** -959) & (np.abs(x) < 2.0 ** 959)
    assert units(np.ascontiguousarray(rcp[reach])).max() <= 1 and units(np.ascontiguousarray(rcp[~reach])).max() == 0
    reach &= x > 0
    assert units(np.ascontiguousarray(root[reach])).max() <= 1 and units(np.ascontiguousarray(root[~reach])).max() == 0
    mid = (np.abs(x) < 2.0 ** 900) & ((np.abs(x) > 2.0 ** -900) | (x == 0.0))
    for v in divs:
        assert units(np.ascontiguousarray(v[mid])).max() == 0


def test_float_to_double_by_bits(arith):
    """All 2^32 patterns."""
    import torch

    bad = torch.zeros(2, dtype=torch.int32, device="cuda")
    arith("arith_f2d", bad)
    assert bad.tolist() == [0, 0]


BPADE = 1.0 / 0.278


def test_fp64_table_index(arith):
    """The nearest integer of 10000 ze / (bpade + ze), or its neighbour where the
    quotient is within 1e-11 (four roundings of a number below 10,000) of a half."""
    import torch

    arith("arith_sw_table", C.c_double(BPADE))
    rng = np.random.default_rng(4)
    ze = 10.0 ** rng.uniform(np.log10(0.06), 18.0, 1 << 18)
    ze[: 1 << 17] = rng.uniform(0.06, 500.0, 1 << 17)
    d = torch.from_numpy(ze).cuda()
    itr = torch.empty(d.numel(), dtype=torch.int32, device="cuda")
    arith("arith_index64", d, itr, C.c_longlong(d.numel()))
    z = ze.astype(np.longdouble)
    x = 10000 * z / (np.longdouble(BPADE) + z)
    assert (np.abs(itr.cpu().numpy() - x) <= 0.5 + 1e-11).all()


@pytest.mark.parametrize("total", [0, 1])
def test_reftra_fast_divisions(arith, total):
    """The layer solution with div_mid and the table read without branches against
    the operators: the same values (signed zeros and results below 1e-37 aside)
    over what the guard lets through -- optical depths of 2^-84 (2^-60 scaled by
    1 - omega g^2) to 2^60, every sun, albedo and asymmetry, the delta-scaled
    asymmetries g / (1 + g) near -1 and 1 too -- and not a number in the same places."""
    import torch

    n = 1 << 21
    rng = np.random.default_rng(11 + total)
    pick = lambda p: rng.random(n) < p
    mu = np.where(pick(0.5), rng.uniform(0.01, 1.0, n), 10.0 ** rng.uniform(-10.0, 0.0, n))
    tau = np.where(pick(0.5), 10.0 ** rng.uniform(-6.0, 3.0, n), 2.0 ** rng.uniform(-84.0, 60.0, n))
    zco = np.where(pick(0.5), rng.uniform(0.0, 1.0, n), 10.0 ** rng.uniform(-9.0, 0.0, n))
    zco[pick(0.01)] = 0.0
    g = rng.uniform(-1.0, 0.99999, n)
    g[: n // 16] = -1.0 + 2.0 ** rng.uniform(-24.0, 0.0, n // 16)
    zg = np.where(pick(0.7), g / (1.0 + g), rng.uniform(0.0, 1.0, n))
    zg[pick(0.01)], zg[pick(0.01)] = 0.0, 1.0
    f = lambda v: torch.from_numpy(np.asarray(v, dtype=np.float32)).cuda()
    zw = np.float32(1.0) - zco.astype(np.float32)
    i = np.arange(10001) / 10000.0
    with np.errstate(divide="ignore"):
        tab = np.exp(-BPADE * i / (1.0 - i))
    tab[10000] = 1e-20
    arith("arith_sw_table", C.c_double(BPADE))
    out = torch.empty((2, n, 5), dtype=torch.float32, device="cuda")
    arith("arith_reftra", f(tab), f(zg), f(mu), f(tau), f(zw), f(zco), out, total, C.c_longlong(n))
    a, b = out[0].double(), out[1].double()
    same = (a == b) | (a.isnan() & b.isnan()) | ((a - b).abs() <= 1e-37)
    where = torch.nonzero(~same.all(1)).flatten()[:3].tolist()
    assert same.all(), [(zg[k], mu[k], tau[k], zco[k], out[:, k].tolist()) for k in where]
    assert a.isfinite().double().mean() > 0.98
