"""GPU: several element types, the engine's kernel against the general path.

The engine forms Y and the energies together on shared products (k_snap_y_me),
using the inversion symmetry of its own U; the cpuSnap.h stages read any U and
form every layer's products (k_snap_yi_me, k_snap_ei_me).  Two to four elements
with chemflag, every 2J, flags on and off, atom counts around a tile's 32 and
above one wave of CTAs: energies within 1e-12 and forces and the total virial
within 1e-10 of the largest entry, as for the fixtures.
"""
import numpy as np
import pytest

import julia_abi
from mdp_b200 import _lib, configs
from oracle import oracle

pytestmark = pytest.mark.gpu

RAD, WJ = (0.5, 0.46, 0.48, 0.44), (1.0, 0.93, 0.9, 0.8)
CASES = [(2, 4, (2, 2, 2), {}), (2, 8, (2, 2, 4), dict(wselfallflag=1)), (3, 6, (3, 3, 3), dict(bnormflag=1, bzeroflag=1)),
         (4, 4, (4, 4, 4), dict(bzeroflag=1)), (4, 6, (3, 3, 4), {}), (4, 8, (2, 2, 4), dict(bnormflag=1)),
         (2, 6, (11, 10, 11), {}), (3, 4, (11, 11, 12), dict(wselfallflag=1, bzeroflag=1))]


def rel_inf(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("ne,tj,cells,flags", CASES)
@pytest.mark.parametrize("vac", [0, 1])
def test_engine_equals_the_stages(cuda_lib, ne, tj, cells, flags, vac):
    from mdp_b200.snap import snap_compute
    p = configs.snap_params_elements(tj, RAD[:ne], WJ[:ne], chemflag=1, seed=31, **flags)
    cfg = configs.ta_config(cells, temp=0.0, jitter=0.07, seed=6)
    x = np.ascontiguousarray(cfg.x[vac:])
    n = x.shape[0]
    types = np.random.default_rng(ne).integers(1, ne + 1, n).astype(np.int32)
    xa, al, nl, nn = oracle.neighbor_list(x, cfg.box, p.rcut, 1.0, 80)
    g = dict(x=x, xall=xa, alist=al, neighlist=nl, neighnum=nn, types=types)
    want = julia_abi.snap_sequence_elements(julia_abi.bind(_lib.LIB_PATH), g, p)
    out = snap_compute(p, x, cfg.box, 1.0, 80, types=types)
    assert rel_inf(out["eatom"], want["eatom"]) < 1e-12
    assert rel_inf(out["fatom"], want["fatom"].reshape(n, 3)) < 1e-10
    assert rel_inf(out["vatom"].sum(1), want["vatom"].reshape(n, 6).sum(0)) < 1e-10
