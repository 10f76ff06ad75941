"""GPU: the cpuSnap.h stages against the repository's own oracle and fixtures.

The same call sequences that are compared with MDP's built CPU library where that
is at hand, here against the C oracle (U, B, Y, energies, forces, total virial)
and, for several element types, against the fixtures of MDP's force chain; and Y
of a U that lacks the inversion symmetry, whose right-hand rows must be read as
given.  FP64: 1e-12 of the largest entry for U and energies, 1e-10 for what is
contracted from them, as in the comparison with MDP's library.
"""
import numpy as np
import pytest

import julia_abi
from conftest import golden_params, load_golden
from mdp_b200 import _lib, configs
from oracle import oracle

pytestmark = pytest.mark.gpu


def rel_inf(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("name", ["bcc128_2j4", "bcc128_2j6", "bcc250_2j8", "bcc250_2j8_hot", "bcc54_2j8_flags"])
def test_stages_match_oracle(cuda_lib, name):
    g = load_golden(name)
    p = golden_params(g)
    e, f, v, U, Y, B = oracle.snap_force(g["xall"], g["alist"], g["neighlist"], g["neighnum"], p, want_uy=True)
    b = julia_abi.snap_sequence(julia_abi.bind(_lib.LIB_PATH), g, p)
    n = g["x"].shape[0]
    for k in (0, 1):
        assert rel_inf(b["u"][k].reshape(-1, n).T, U[:, k]) < 1e-12
        assert rel_inf(b["y"][k].reshape(-1, n).T, Y[:, k]) < 1e-10
    assert rel_inf(b["eatom"], e) < 1e-12
    assert rel_inf(b["blist"].reshape(-1, n).T, B) < 1e-10
    assert rel_inf(b["fatom"].reshape(n, 3), f) < 1e-10
    # the Julia layout books a pair's virial on its first atom, the core on both
    assert rel_inf(b["vatom"].reshape(n, 6).sum(0), v.sum(1)) < 1e-10


@pytest.mark.parametrize("name", ["chem_bcc128_2j6", "chem_bcc250_2j8", "chem_bcc54_2j4_3el_flags",
                                  "chem_bcc54_2j6_wselfall"])
def test_stages_of_several_elements_match_fixtures(cuda_lib, name):
    g = load_golden(name)
    bnorm, bzero, switch, wsa = (int(v) for v in g["flags"])
    p = configs.snap_params_elements(int(g["twojmax"]), g["radelems"], g["wjelems"], chemflag=int(g["chemflag"]),
                                     seed=int(g["coeff_seed"]), bnormflag=bnorm, bzeroflag=bzero,
                                     switchflag=switch, wselfallflag=wsa)
    b = julia_abi.snap_sequence_elements(julia_abi.bind(_lib.LIB_PATH), g, p)
    n = g["x"].shape[0]
    assert rel_inf(b["eatom"], g["eatom"]) < 1e-12
    assert rel_inf(b["fatom"].reshape(n, 3), g["fatom"]) < 1e-10
    assert rel_inf(b["vatom"].reshape(n, 6).sum(0), g["vatom"].sum(1)) < 1e-10


def y_of(U, p):
    """Y rows mb <= j/2 of full-plane U (n, nu), every entry read as given
    (cpuSnapComputeYi of one element, cpuSnap4.cpp:697-792)."""
    tj = p.twojmax
    t = oracle.tables(tj)
    cgb, k = {}, 0
    for j1 in range(tj + 1):
        for j2 in range(j1 + 1):
            for j in range(j1 - j2, min(tj, j1 + j2) + 1, 2):
                cgb[j1, j2, j] = k
                k += (j1 + 1) * (j2 + 1)
    kb = {tuple(int(v) for v in q): i for i, q in enumerate(t["idxb"])}
    ub = t["idxu_block"]
    Y = np.zeros_like(U)
    for j1, j2, j, a1, a2, na, b1, b2, nb, u in ((int(v) for v in q) for q in t["idxz"]):
        if j >= j1:
            beta = p.coeff[1 + kb[j1, j2, j]] * ((3.0 if j2 == j else 2.0) if j1 == j else 1.0)
        elif j >= j2:
            beta = p.coeff[1 + kb[j, j2, j1]] * (2.0 if j2 == j else 1.0)
        else:
            beta = p.coeff[1 + kb[j2, j, j1]]
        if p.bnormflag:
            beta /= j + 1
        elif j1 > j:
            beta *= (j1 + 1) / (j + 1.0)
        c = t["cg"][cgb[j1, j2, j]:][: (j1 + 1) * (j2 + 1)].reshape(j1 + 1, j2 + 1)
        z = 0.0
        for ib in range(nb):
            r1 = U[:, ub[j1] + (j1 + 1) * (b1 + ib):][:, : j1 + 1]
            r2 = U[:, ub[j2] + (j2 + 1) * (b2 - ib):][:, : j2 + 1]
            z = z + c[b1 + ib, b2 - ib] * sum(c[a1 + ia, a2 - ia] * r1[:, a1 + ia] * r2[:, a2 - ia] for ia in range(na))
        Y[:, u] += beta * z
    return Y


@pytest.mark.parametrize("tj,n,bnorm", [(4, 33, 0), (6, 5, 1), (8, 32, 0)])
def test_y_of_any_u(cuda_lib, tj, n, bnorm):
    p = configs.snap_params(tj, seed=4, bnormflag=bnorm)
    L = julia_abi.bind(_lib.LIB_PATH)
    t = julia_abi.tables(L, tj)
    rng = np.random.default_rng(tj)
    U = rng.normal(size=(n, t["nu"])) + 1j * rng.normal(size=(n, t["nu"]))
    want = y_of(U, p)
    ur, ui = (np.ascontiguousarray(a.T).ravel() for a in (U.real, U.imag))
    yr = np.zeros(n * t["nu"]); yi = np.zeros(n * t["nu"])
    coeff = np.ascontiguousarray(p.coeff)
    one = np.ones(n, dtype=np.int32); mp = np.zeros(2, dtype=np.int32)
    L.cpuSnapComputeYi(yr, yi, ur, ui, t["cg"], coeff, mp, one, t["idxz"], t["idxb_block"], t["idxu_block"],
                       t["idxcg_block"], tj, t["nb"], t["nu"], t["nz"], 1, coeff.size, bnorm, 0, n)
    got = (yr + 1j * yi).reshape(t["nu"], n).T
    assert rel_inf(got, want) < 1e-12
