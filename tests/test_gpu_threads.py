"""Host threads with a context each: calls of different sizes, layers and kinds
at the same time (what a kernel is launched with must not depend on what
another thread asked for in between)."""
import threading

import numpy as np
import pytest

from brams_gb300 import rrtmg_lw as R
from test_gpu_capture import Batch, Dropin, Nomcica, Shortwave, _direct

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kinds", [(Dropin, Dropin), (Batch, Nomcica), (Shortwave, Batch)])
def test_calls_of_two_threads(kinds):
    import torch

    ctxs = [R.Context() for _ in kinds]
    calls = [k(c, n) for k, c, n in zip(kinds, ctxs, (40, 700))]
    refs = [_direct(c) for c in calls]
    streams = [torch.cuda.Stream() for _ in calls]
    torch.cuda.synchronize()
    errors = []

    def work(c, s):
        try:
            for _ in range(2000):
                c.run(s.cuda_stream)
            s.synchronize()
        except Exception as e:  # a launch that was refused
            errors.append(e)

    threads = [threading.Thread(target=work, args=(c, s)) for c, s in zip(calls, streams)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors[0]
    for c, ref in zip(calls, refs):
        assert c.ctx.sync_status() == 0
        for k, v in ref.items():
            assert np.array_equal(c.d[k].cpu().numpy(), v), k
        c.ctx.close()
