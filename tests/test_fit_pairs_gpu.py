"""GPU: pair search of the batched fit, atoms a lane each.

Configurations of 1, 31, 32, 33, 64 and 65 atoms, none of whose atoms have a
pair, some have, and each has more than the 32 pairs that are emitted at a time
from 32 atoms; in one batch and each alone.  Pair counts against a count by
numpy, per-atom B against the oracle (FP64, 1e-12 of the largest entry: sums of
some 1e5 terms at 1e-16, with random signs).
"""
import itertools
import time

import numpy as np
import pytest

from mdp_b200 import configs
from mdp_b200.fit import BatchFit, FitConfig
from oracle import oracle

pytestmark = pytest.mark.gpu


def gas(n, edge, seed):
    """n atoms at random, no two (nor images) closer than 1 A."""
    rng = np.random.default_rng(seed)
    x = np.zeros((0, 3))
    while x.shape[0] < n:
        y = edge * rng.random(3)
        d = x - y
        d -= edge * np.round(d / edge)
        if (d * d).sum(1).min(initial=9.0) > 1.0:
            x = np.vstack([x, y])
    return FitConfig(x=x, box=np.full(3, edge), kind="gas")


def npairs(c, rcut):
    sh = np.array(list(itertools.product((-1, 0, 1), repeat=3))) * c.box
    d = c.x[None, :, None] + sh[None, None] - c.x[:, None, None]
    r2 = (d * d).sum(-1)
    return int(((r2 < rcut * rcut) & (r2 > 1e-20)).sum())


CASES = [(1, 30.0), (31, 40.0), (31, 9.0), (32, 9.0), (33, 9.0), (33, 6.0), (64, 6.5), (65, 7.0), (65, 30.0)]


def test_pairs_and_descriptors_at_the_edges(cuda_lib):
    p = configs.snap_params(4, seed=3)
    cfgs = [gas(n, edge, 10 + k) for k, (n, edge) in enumerate(CASES)]
    want = [npairs(c, p.rcut) for c in cfgs]
    assert want[0] == 0 and max(w / c.natoms for w, c in zip(want, cfgs)) > 64
    bf = BatchFit(p)
    bf.set_batch(cfgs)
    assert bf.npairs() == sum(want)
    _, bd, _, bl = bf.descriptors()
    a0 = 0
    for c, w in zip(cfgs, want):
        n = c.natoms
        xa, al, nl, nn = oracle.neighbor_list(c.x, c.box, p.rcut, 0.0, 512)
        B = oracle.snap_force(xa, al, nl, nn, p, want_uy=True)[5]
        assert np.abs(bl[:, a0:a0 + n].T - B).max() < 1e-12 * np.abs(B).max()
        one = BatchFit(p)
        one.set_batch([c])
        assert one.npairs() == w
        _, d1, _, b1 = one.descriptors()
        assert np.array_equal(b1, bl[:, a0:a0 + n]) and np.array_equal(d1, bd[a0:a0 + n])
        one.close()
        a0 += n
    bf.close()


def test_large_cells_are_searched_quickly(cuda_lib):
    """20 configurations of 2,048 atoms, 2.3e9 candidates in each of the two passes:
    4.4 ms in all.  A kernel that takes atom and image apart from each candidate's
    number spends 13 ms, one of a thread per atom 12."""
    cfgs = []
    for k in range(20):
        x, box = configs.lattice((8, 8, 8), "fcc", 4.2)
        x = np.mod(x + np.random.default_rng(k).normal(0.0, 0.03, x.shape), box)
        cfgs.append(FitConfig(x=np.where(x >= box, x - box, x), box=box, kind="fcc"))
    bf = BatchFit(configs.snap_params(4, seed=3))
    t = []
    for _ in range(8):
        a = time.perf_counter()
        bf.set_batch(cfgs)
        t.append(time.perf_counter() - a)
    bf.close()
    assert min(t) < 8e-3, t
