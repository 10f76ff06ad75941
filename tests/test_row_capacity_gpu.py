"""GPU: neighbour rows of a caller that have far more slots than entries.

The results do not depend on the rows' capacity, bit for bit, and the time of a
call goes with the entries: 128,000 atoms take the same time with rows of 64 and
of 1,000 slots (1.04 ms each; a kernel that touches every slot takes 1.6 times
as long, so the limit of 1.3 lies between).
"""
import ctypes as C

import numpy as np
import pytest

from mdp_b200 import _lib, configs
from oracle import oracle

pytestmark = pytest.mark.gpu


def caller(lib, p, lists, nm):
    """(call, outputs) of mdp_snap_compute_device on rows of nm slots."""
    import torch
    xa, al, nl, nn = lists
    n = nl.shape[0]
    rows = np.zeros((n, nm), dtype=np.int32)
    rows[:, :64] = nl
    t = [torch.from_numpy(np.ascontiguousarray(a, dtype=d)).cuda()
         for a, d in ((xa, np.float64), (al, np.int32), (rows, np.int32), (nn, np.int32))]
    sp, keep = _lib.snap_params_c(p)
    out = torch.empty(10 * n, dtype=torch.float64, device="cuda")
    at = lambda k: out.data_ptr() + 8 * k * n

    def call(held=(t, keep)):
        _lib.check(lib.mdp_snap_compute_device(C.byref(sp), 0, *[a.data_ptr() for a in held[0]], n, xa.shape[0], nm,
                                               at(0), at(1), at(4),
                                               C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return call, out


@pytest.mark.parametrize("nm", [64, 65, 96, 1000])
def test_results_do_not_depend_on_the_capacity(cuda_lib, nm):
    import torch
    p = configs.snap_params(6, seed=11)
    cfg = configs.ta_config((5, 5, 6), temp=0.0, jitter=0.07, seed=2)
    lists = oracle.neighbor_list(cfg.x, cfg.box, p.rcut, 1.0, 64)
    want_call, want = caller(cuda_lib, p, lists, 64)
    call, out = caller(cuda_lib, p, lists, nm)
    want_call()
    call()
    torch.cuda.synchronize()
    assert torch.equal(out, want)


def test_time_goes_with_the_entries(cuda_lib):
    import torch
    p = configs.snap_params(4, seed=11)
    cfg = configs.ta_config((40, 40, 40), temp=0.0, jitter=0.07, seed=2)
    lists = oracle.neighbor_list(cfg.x, cfg.box, p.rcut, 1.0, 64)
    ms = []
    for nm in (64, 1000):
        call, _ = caller(cuda_lib, p, lists, nm)
        t = []
        for _ in range(25):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            call()
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b))
        ms.append(min(t[5:]))
    assert ms[1] < 1.3 * ms[0], ms
