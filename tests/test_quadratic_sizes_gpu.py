"""GPU: quadratic SNAP at the sizes where the Y kernel's work split changes.

Y with per-atom coefficients takes the branches of the linear model (couplings
shared by up to eight groups, one group, a last wave of its own), each with its
own offsets into the coefficients.  A cell that the many-group branch evaluates,
the one that MDP's fixtures cover, is repeated until the others do: every copy
has the cell's energies, forces and virials.  A force is the product of two sums
of some 4e4 terms at 1e-16 with random signs, and a copy's coordinates carry the
rounding of the box they lie in: 2e-12, or 6e-14 per A of the box, of the largest
entry.  With Q = 0 the model is a linear one: within 1e-12 of the oracle.
"""
import numpy as np
import pytest

from mdp_b200 import configs
from oracle import oracle

pytestmark = pytest.mark.gpu


def crystal(cells, vac, seed):
    cfg = configs.ta_config(cells, temp=0.0, jitter=0.07, seed=seed)
    keep = np.ones(cfg.natoms, dtype=bool)
    keep[np.random.default_rng(seed).choice(cfg.natoms, vac, replace=False)] = False
    return np.ascontiguousarray(cfg.x[keep]), cfg.box


@pytest.mark.parametrize("tj", [4, 6, 8])
@pytest.mark.parametrize("reps,tiles", [((3, 3, 3), 108), ((4, 4, 3), 191), ((5, 5, 4), 397)])
def test_copies_of_a_cell(cuda_lib, reps, tiles, tj):
    from mdp_b200.snap import snap_compute
    p = configs.snap_params(tj, seed=11, quadraticflag=1)
    x, box = crystal((4, 4, 4), 1, 5)
    want = snap_compute(p, x, box, 1.0, 80)
    i = np.stack(np.meshgrid(*[np.arange(r) for r in reps], indexing="ij"), -1).reshape(-1, 1, 3)
    xs, boxs = np.ascontiguousarray((x[None] + i * box).reshape(-1, 3)), box * np.asarray(reps)
    assert (xs.shape[0] + 31) // 32 == tiles
    out = snap_compute(p, xs, boxs, 1.0, 80)
    tol = max(2e-12, 6e-14 * max(boxs))
    for k in ("eatom", "fatom", "vatom"):
        got, ref = (a[k].T if k == "vatom" else a[k] for a in (out, want))
        ref = np.tile(ref, (np.prod(reps),) + (1,) * (ref.ndim - 1))
        assert np.abs(got - ref).max() < tol * np.abs(ref).max()


@pytest.mark.parametrize("tj", [6, 8])
@pytest.mark.parametrize("cells,vac", [((2, 2, 3), 1), ((9, 9, 9), 2), ((10, 11, 11), 37), ((14, 14, 13), 40)])
def test_without_quadratic_terms(cuda_lib, cells, vac, tj):
    from mdp_b200.snap import snap_compute
    lin = configs.snap_params(tj, seed=11)
    p = configs.snap_params(tj, seed=11, quadraticflag=1, qsigma=0.0)
    assert np.array_equal(p.coeff[: lin.coeff.size], lin.coeff) and not p.coeff[lin.coeff.size:].any()
    x, box = crystal(cells, vac, 5)
    xa, al, nl, nn = oracle.neighbor_list(x, box, lin.rcut, 1.0, 80)
    want = oracle.snap_force(xa, al, nl, nn, lin)
    out = snap_compute(p, x, box, 1.0, 80)
    for k, ref in zip(("eatom", "fatom", "vatom"), want):
        assert np.abs(out[k] - ref).max() < 1e-12 * np.abs(ref).max()
