"""GPU: force stages at the sizes where their work split changes.

The Y kernel gives a tile's couplings to one CTA or shares them among up to
eight (few tiles, or few in the last wave), and its FP32 form puts two tiles in
a CTA; ragged atom counts leave lanes, or a CTA's second tile, empty.  The U
kernel gives an atom's pairs to four lanes (few tiles) or one.  Energies, forces and
virials against the oracle: FP64 within 1e-12 of the largest entry (sums of
about 4e4 terms at 1e-16 each, some 2e-14 with random signs, times the
cancellation of a force sum), FP32 forces within 1e-5 of it.
"""
import numpy as np
import pytest

from mdp_b200 import configs
from oracle import oracle

pytestmark = pytest.mark.gpu

SIZES = [
    ((2, 2, 2), 0),       # half a tile, eight groups
    ((2, 2, 3), 1),
    ((4, 4, 1 + 3), 0),   # four full tiles
    ((4, 4, 5), 31),      # five tiles less 31 atoms: 129 atoms
    ((9, 9, 9), 2),       # three groups (FP64)
    ((10, 11, 11), 37),   # 75 tiles: one group (FP64), the FP32 CTA's second tile missing
    ((14, 14, 13), 40),   # 158 tiles: one group, FP64's last ten tiles a wave of their own
    ((17, 17, 17), 3),    # 307 tiles: the same in FP32
]


def crystal(cells, vac, seed):
    cfg = configs.ta_config(cells, temp=0.0, jitter=0.07, seed=seed)
    keep = np.ones(cfg.natoms, dtype=bool)
    keep[np.random.default_rng(seed).choice(cfg.natoms, vac, replace=False)] = False
    return np.ascontiguousarray(cfg.x[keep]), cfg.box


def rel(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("tj", [4, 6, 8])
@pytest.mark.parametrize("cells,vac", SIZES)
def test_force_stages_match_oracle(cuda_lib, cells, vac, tj):
    from mdp_b200.snap import snap_compute
    if tj != 8 and np.prod(cells) > 1000:
        pytest.skip("the largest sizes are covered at 2J = 8")
    p = configs.snap_params(tj, seed=11)
    x, box = crystal(cells, vac, 5)
    xa, al, nl, nn = oracle.neighbor_list(x, box, p.rcut, 1.0, 80)
    e, f, v = oracle.snap_force(xa, al, nl, nn, p)
    out = snap_compute(p, x, box, 1.0, 80)
    assert rel(out["eatom"], e) < 1e-12 and rel(out["fatom"], f) < 1e-12 and rel(out["vatom"], v) < 1e-12
    out = snap_compute(p, x, box, 1.0, 80, precision="fp32")
    assert rel(out["eatom"], e) < 1e-6 and rel(out["fatom"], f) < 1e-5 and rel(out["vatom"], v) < 1e-5


@pytest.mark.parametrize("cells,vac,jitter", [((2, 2, 2), 0, 0.0), ((3, 3, 4), 3, 0.25), ((6, 6, 6), 0, 0.1)])
def test_neighbour_rows_at_their_capacity(cuda_lib, cells, vac, jitter):
    """Rows that the fullest atom fills exactly (powers of two and not) equal the
    oracle's index for index; one slot less is an error."""
    from mdp_b200 import _lib
    from mdp_b200.snap import snap_compute
    p = configs.snap_params(4, seed=11)
    cfg = configs.ta_config(cells, temp=0.0, jitter=jitter, seed=9)
    keep = np.ones(cfg.natoms, dtype=bool)
    keep[:vac] = False
    x = np.ascontiguousarray(cfg.x[keep])
    for skin in (0.2, 1.0):
        xa, al, nl, nn = oracle.neighbor_list(x, cfg.box, p.rcut, skin, 128)
        nm = int(nn.max())
        out = snap_compute(p, x, cfg.box, skin, nm, want_neighbors=True)
        assert np.array_equal(out["neighnum"], nn)
        for i in range(x.shape[0]):
            assert np.array_equal(out["neighlist"][i, :nn[i]], np.sort(nl[i, :nn[i]]))
        with pytest.raises(_lib.MdpError, match="overflow"):
            snap_compute(p, x, cfg.box, skin, nm - 1)


@pytest.mark.parametrize("nm", [3072, 3073, 5000])
def test_long_neighbour_rows(cuda_lib, nm):
    """Rows longer than a warp's shared memory holds are collected and sorted in place."""
    from mdp_b200.snap import snap_compute
    p = configs.snap_params(4, seed=11)
    x, box = crystal((3, 3, 4), 2, 7)
    want = snap_compute(p, x, box, 1.0, 128, want_neighbors=True)
    out = snap_compute(p, x, box, 1.0, nm, want_neighbors=True)
    assert np.array_equal(out["neighnum"], want["neighnum"])
    for i, n in enumerate(want["neighnum"]):
        assert np.array_equal(out["neighlist"][i, :n], want["neighlist"][i, :n])
    assert np.array_equal(out["fatom"], want["fatom"])


def replicate(x, box, reps):
    """reps copies of a cell along its axes; the copies of an atom stay apart by n."""
    i = np.stack(np.meshgrid(*[np.arange(r) for r in reps], indexing="ij"), -1).reshape(-1, 1, 3)
    return np.ascontiguousarray((x[None] + i * box).reshape(-1, 3)), box * np.asarray(reps)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("kind,reps,tj", [("crystal", (8, 8, 7), 8), ("crystal", (10, 8, 10), 6), ("gas", (17, 16, 16), 8)])
def test_large_systems_repeat_their_cell(cuda_lib, kind, reps, tj, precision):
    """Above the size from which dE/dr runs as one sweep: a cell repeated to more
    than 49,152 (2J = 6 FP32: 98,304) atoms has the cell's energies, forces and
    virials in every copy.  The gas, a pair or two per atom, makes a window of
    pairs span several turns of staged atoms, with pairless atoms between."""
    from mdp_b200.snap import snap_compute
    p = configs.snap_params(tj, seed=11)
    if kind == "crystal":
        x, box = crystal((4, 4, 4), 1, 5)
    else:
        rng = np.random.default_rng(3)
        box = np.full(3, 13.0)
        x = box * rng.random((12, 3))
    xa, al, nl, nn = oracle.neighbor_list(x, box, p.rcut, 1.0, 80)
    want = oracle.snap_force(xa, al, nl, nn, p)
    xs, boxs = replicate(x, box, reps)
    assert xs.shape[0] > (98304 if tj == 6 else 49152)
    out = snap_compute(p, xs, boxs, 1.0, 80, precision=precision)
    tol = 1e-12 if precision == "fp64" else 1e-5
    # coordinates of a copy carry the rounding of the box they lie in
    tol = max(tol, 1e-15 * max(boxs) * 30)
    for got, ref in zip((out["eatom"], out["fatom"], out["vatom"].T), (want[0], want[1], want[2].T)):
        ref = np.tile(ref, (xs.shape[0] // x.shape[0],) + (1,) * (ref.ndim - 1))
        assert np.abs(got - ref).max() < tol * np.abs(ref).max()
