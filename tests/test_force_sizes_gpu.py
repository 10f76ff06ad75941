"""GPU: force stages at the sizes where their work split changes.

The Y kernel gives a tile's couplings to one CTA or shares them among up to
eight (few tiles), and its FP32 form puts two tiles in a CTA; ragged atom
counts leave lanes, or a CTA's second tile, empty.  Energies, forces and
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
    ((14, 14, 13), 40),   # 158 tiles: one group in both precisions
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
