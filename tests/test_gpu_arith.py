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
