"""GPU: a force call captured into a graph after a larger system has been evaluated.

The work buffers of a process have their size after the largest system's call, so
a smaller one can be captured, whichever split of the Y kernel it takes.  Each
model in a process of its own, whose first call is the larger one.
"""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SCRIPT = """
import ctypes as C, sys
import numpy as np, torch
from mdp_b200 import _lib, configs
from oracle import oracle
tj, prec, quad = (int(a) for a in sys.argv[1:])
L = _lib.lib()
p = configs.snap_params(tj, seed=1, quadraticflag=quad)
sp, keep = _lib.snap_params_c(p)
stream = torch.cuda.Stream()

def system(cells):
    cfg = configs.ta_config(cells, temp=0.0, jitter=0.07, seed=1)
    xa, al, nl, nn = oracle.neighbor_list(cfg.x, cfg.box, p.rcut, 1.0, 64)
    t = [torch.from_numpy(np.ascontiguousarray(a, dtype=d)).cuda()
         for a, d in ((xa, np.float64), (al, np.int32), (nl, np.int32), (nn, np.int32))]
    n = cfg.natoms
    def call():
        with torch.cuda.stream(stream):
            o = torch.zeros(10 * n, dtype=torch.float64, device="cuda")
            at = lambda k: o.data_ptr() + 8 * k * n
            _lib.check(L.mdp_snap_compute_device(C.byref(sp), prec, *[a.data_ptr() for a in t], n, xa.shape[0], 64,
                                                 at(0), at(1), at(4), C.c_void_p(stream.cuda_stream)))
        return o
    return call

small = [system(c) for c in ((2, 2, 2), (5, 5, 5), (9, 9, 9))]
system((12, 12, 12))()          # 108 tiles: couplings not shared
torch.cuda.synchronize()
for call in small:
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream):
        o = call()
    g.replay()
    torch.cuda.synchronize()
    want = call()
    torch.cuda.synchronize()
    assert torch.isfinite(want).all() and torch.equal(o, want)
print("same")
"""


@pytest.mark.parametrize("tj,prec,quad", [(8, 0, 0), (6, 0, 0), (8, 1, 0), (6, 1, 0), (8, 0, 1), (4, 0, 0)])
def test_smaller_systems_can_be_captured(cuda_lib, tj, prec, quad):
    r = subprocess.run([sys.executable, "-c", SCRIPT, str(tj), str(prec), str(quad)], cwd=ROOT, capture_output=True,
                       text=True, timeout=300, env=dict(os.environ, PYTHONPATH=ROOT))
    assert r.returncode == 0 and "same" in r.stdout, r.stderr[-2000:]
