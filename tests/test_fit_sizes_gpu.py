"""GPU: the batched descriptors on configurations of few and of many pairs.

The batch's pairs are emitted 32 at a time, its reverse lists sorted by rank up
to 128 entries and in place beyond, and a configuration's sums shared by sixteen
threads: cells from no pair to more than 128 pairs per atom, in one batch.
Against the oracle through a linear model: the per-atom B; E = beta . B summed,
f = bd beta and the total virial, FP64 within 1e-12 of the largest entry (sums
of some 1e5 terms at 1e-16, with random signs).
"""
import numpy as np
import pytest

from mdp_b200 import configs
from mdp_b200.fit import FitConfig
from oracle import oracle

pytestmark = pytest.mark.gpu


def fcc(n, a, jitter, seed):
    x, box = configs.lattice((n, n, n), "fcc", a)
    x = np.mod(x + np.random.default_rng(seed).normal(0.0, jitter, x.shape), box)
    return FitConfig(x=np.where(x >= box, x - box, x), box=box, kind="fcc")


@pytest.mark.parametrize("tj", [4, 6, 8])
def test_descriptors_of_sparse_and_dense_cells(cuda_lib, tj):
    from mdp_b200.fit import BatchFit
    rng = np.random.default_rng(1)
    p = configs.snap_params(tj, seed=3)
    cfgs = [FitConfig(x=np.full((1, 3), 1.0), box=np.full(3, 9.0), kind="one"),          # no pair
            FitConfig(x=9.0 * rng.random((5, 3)), box=np.full(3, 9.0), kind="gas"),
            fcc(2, 4.2, 0.05, 2),      # 18 pairs per atom or so
            fcc(2, 3.3, 0.05, 3),      # above 32
            fcc(3, 2.6, 0.03, 4),      # above 64
            fcc(3, 2.1, 0.02, 5)]      # above 128
    bf = BatchFit(p)
    bf.set_batch(cfgs)
    bi, bd, bv, bl = bf.descriptors()
    beta, a0, most = p.coeff[1:], 0, 0
    for c, cfg in enumerate(cfgs):
        n = cfg.natoms
        xa, al, nl, nn = oracle.neighbor_list(cfg.x, cfg.box, p.rcut, 0.0, 512)
        most = max(most, int(nn.max()))
        e, f, v, _, _, B = oracle.snap_force(xa, al, nl, nn, p, want_uy=True)
        scale = lambda t: max(np.abs(t).max(), 1e-3)
        assert np.abs(bl[:, a0:a0 + n].T - B).max() < 1e-12 * scale(B)
        assert np.abs(bi[c] - B.sum(0)).max() < 1e-12 * scale(B.sum(0))
        assert abs(bi[c] @ beta + n * p.coeff[0] - e.sum()) < 1e-12 * scale(e.sum())
        terms = np.abs(bd[a0:a0 + n]).max() * np.abs(beta).sum()   # the size of what cancels in a force
        assert np.abs(bd[a0:a0 + n] @ beta - f).max() < 1e-12 * max(terms, 1e-3)
        tv = np.abs(bv[c]).max() * np.abs(beta).sum()
        assert np.abs(beta @ bv[c] - v.sum(1)).max() < 1e-12 * max(tv, 1e-3)
        a0 += n
    assert most > 128
