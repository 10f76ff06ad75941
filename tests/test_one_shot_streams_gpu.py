"""GPU: force calls on several streams and threads.

`mdp_snap_compute_device` returns when its work is queued, and all calls of a
device share their work buffers.  Systems of different sizes, models and
precisions are evaluated in turn on streams that nothing else orders, from one
thread and from several; each result equals the one of a call by itself bit for
bit (every sum has a fixed order).
"""
import ctypes as C
import threading

import numpy as np
import pytest

from mdp_b200 import _lib, configs
from oracle import oracle

pytestmark = pytest.mark.gpu

NM = 80
# cells, vacancies, 2J, precision, options: a long call beside short ones
SYSTEMS = [((16, 16, 15), 5, 8, 0, {}), ((2, 2, 3), 1, 8, 0, {}), ((4, 4, 4), 0, 6, 1, {}),
           ((5, 5, 4), 7, 6, 0, dict(quadraticflag=1))]


class System:
    def __init__(self, lib, cells, vac, tj, prec, kw):
        import torch
        p = configs.snap_params(tj, seed=11, **kw)
        cfg = configs.ta_config(cells, temp=0.0, jitter=0.07, seed=vac + tj)
        x = np.ascontiguousarray(cfg.x[vac:])
        xa, al, nl, nn = oracle.neighbor_list(x, cfg.box, p.rcut, 1.0, NM)
        self.sp, self.keep = _lib.snap_params_c(p)
        t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a, dtype=d)).cuda()
        self.x, self.al, self.nl, self.nn = t(xa, np.float64), t(al, np.int32), t(nl, np.int32), t(nn, np.int32)
        self.lib, self.prec, self.n = lib, prec, x.shape[0]

    def call(self, stream):
        """Queues one evaluation on the stream; energies, forces and virials."""
        import torch
        with torch.cuda.stream(stream):
            o = torch.full((10 * self.n,), float("nan"), dtype=torch.float64, device="cuda")
            at = lambda k: o.data_ptr() + 8 * k * self.n
            _lib.check(self.lib.mdp_snap_compute_device(
                C.byref(self.sp), self.prec, self.x.data_ptr(), self.al.data_ptr(), self.nl.data_ptr(),
                self.nn.data_ptr(), self.n, self.x.shape[0], NM, at(0), at(1), at(4), C.c_void_p(stream.cuda_stream)))
        return o


@pytest.fixture(scope="module")
def systems(cuda_lib):
    import torch
    s = [System(cuda_lib, *a) for a in SYSTEMS]
    want = []
    for q in s:
        want.append(q.call(torch.cuda.current_stream()))
        torch.cuda.synchronize()
        assert torch.isfinite(want[-1]).all()
    return s, want


def test_calls_on_several_streams(systems):
    import torch
    s, want = systems
    streams = [torch.cuda.Stream() for _ in s] + [torch.cuda.default_stream()]
    got = []
    for k in range(24):
        q = (0, 1, 0, 2, 3, 1)[k % 6]
        got.append((q, s[q].call(streams[k % len(streams)])))
    torch.cuda.synchronize()
    for q, o in got:
        assert torch.equal(o, want[q])


def test_calls_from_several_threads(systems):
    import torch
    s, want = systems
    got = [[] for _ in s]

    def work(k):
        stream = torch.cuda.Stream()
        for _ in range(8):
            got[k].append(s[k].call(stream))
        stream.synchronize()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(s))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(len(s)):
        assert len(got[k]) == 8 and all(torch.equal(o, want[k]) for o in got[k])


def test_a_captured_call_replays(systems):
    """A call can still be captured once its buffers have their size."""
    import torch
    s, want = systems
    stream = torch.cuda.Stream()
    s[1].call(stream)
    stream.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        o = s[1].call(stream)
    s[2].call(stream)
    torch.cuda.synchronize()
    for _ in range(2):
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(o, want[1])
    after = s[2].call(torch.cuda.current_stream())
    torch.cuda.synchronize()
    assert torch.equal(after, want[2])
