"""GPU: dE/dr as one sweep, over the forms of a model.

From 24,576 to 98,304 atoms on, by type and 2J, dE/dr runs as one sweep and four
sums instead of the reverse sweep.  Switching function off, an inner radius,
neighbour weight and angle factor other than the default, bnorm and bzero, and
the per-atom coefficients of quadratic SNAP: a cell that the reverse sweep
evaluates, itself within 1e-10 of the oracle where that has the form, is repeated
to 56,896 (2J = 6 FP32: 114,300) atoms, and every copy has its energies, forces
and virials.  FP64 sums of some 4e4 terms at 1e-16 with random signs (quadratic:
the product of two), FP32 a few 1e-7 of the largest entry; a copy's coordinates
carry the rounding of the box they lie in.
"""
import numpy as np
import pytest

from mdp_b200 import configs
from oracle import oracle

pytestmark = pytest.mark.gpu

FORMS = [dict(switchflag=0), dict(rmin0=0.6, wjelem=0.8), dict(rfac0=0.85, bnormflag=1, bzeroflag=1),
         dict(quadraticflag=1)]


@pytest.mark.parametrize("tj,precision", [(8, "fp64"), (6, "fp64"), (8, "fp32"), (6, "fp32")])
@pytest.mark.parametrize("form", FORMS, ids=lambda f: "-".join(f))
def test_copies_of_a_cell(cuda_lib, form, tj, precision):
    from mdp_b200.snap import snap_compute
    quad = form.get("quadraticflag", 0)
    if quad and precision == "fp32":
        pytest.skip("quadratic SNAP runs in FP64")
    p = configs.snap_params(tj, seed=11, **form)
    cfg = configs.ta_config((4, 4, 4), temp=0.0, jitter=0.07, seed=5)
    x, box = np.ascontiguousarray(cfg.x[1:]), cfg.box
    want = snap_compute(p, x, box, 1.0, 80)
    if not quad:
        xa, al, nl, nn = oracle.neighbor_list(x, box, p.rcut, 1.0, 80)
        for k, ref in zip(("eatom", "fatom", "vatom"), oracle.snap_force(xa, al, nl, nn, p)):
            assert np.abs(want[k] - ref).max() < 1e-10 * np.abs(ref).max()
    reps = (10, 10, 9) if (tj, precision) == (6, "fp32") else (8, 8, 7)
    assert np.prod(reps) * x.shape[0] > (98304 if (tj, precision) == (6, "fp32") else 49152)
    i = np.stack(np.meshgrid(*[np.arange(r) for r in reps], indexing="ij"), -1).reshape(-1, 1, 3)
    out = snap_compute(p, np.ascontiguousarray((x[None] + i * box).reshape(-1, 3)), box * np.asarray(reps), 1.0, 80,
                       precision=precision)
    tol = max(1e-12, 3e-14 * max(box * np.asarray(reps))) * (2 if quad else 1) if precision == "fp64" else 1e-5
    for k in ("eatom", "fatom", "vatom"):
        got, ref = (a[k].T if k == "vatom" else a[k] for a in (out, want))
        ref = np.tile(ref, (np.prod(reps),) + (1,) * (ref.ndim - 1))
        assert np.abs(got - ref).max() < tol * np.abs(ref).max()
