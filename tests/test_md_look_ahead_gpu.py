"""GPU: a step whose force was queued before its rebuild check was read.

The engine queues the force on the kept neighbour list while the check is under
way, as long as the check before found every atom well inside the limit, and
evaluates again should the list turn out to be due after all.  With a skin that
the fastest atom crosses within a few steps that happens; stage timing turns the
look-ahead off.  Positions, velocities, forces, energies and rebuilds of both runs
are the same bit for bit, thermo rows up to the order of their sums (some 1e3
terms at 1e-16), and the launches show that evaluations were thrown away.
"""
import numpy as np
import pytest

from mdp_b200 import configs
from mdp_b200 import surrogate as su
from mdp_b200.snap import SnapMD, launch_count

pytestmark = pytest.mark.gpu


def trajectory(p, cfg, timed, steps, sur=None, types=None, **kw):
    md = SnapMD(p, cfg.box, cfg.natoms, 0.001, **kw)
    if types is not None:
        md.set_types(types)
    if sur is not None:
        md.set_surrogate(sur, judge_every=7, tol=1e9)   # a judged step never looks ahead
    md.set_state(cfg.x, cfg.v)
    md.setup()
    md.stage_timing(timed)
    before = launch_count()
    th, _ = md.run(steps, thermo_every=5)
    launches = launch_count() - before
    out = md.state()
    rebuilds = md.counters()["rebuilds"]
    md.close()
    return out, th, rebuilds, launches


def compare(p, cfg, **kw):
    got, th, rebuilds, launches = trajectory(p, cfg, False, **kw)
    want, checked_th, checked_rebuilds, checked = trajectory(p, cfg, True, **kw)
    assert rebuilds == checked_rebuilds > 2
    assert launches > checked   # evaluations on a list that was due
    for a, b in zip(got, want):
        assert np.isfinite(a).all() and np.array_equal(a, b)
    assert (np.abs(th - checked_th).max(0) <= 1e-12 * np.abs(th).max(0)).all()


@pytest.mark.parametrize("precision,every,skin", [("fp64", 1, 0.04), ("fp32", 1, 0.04), ("fp64", 4, 0.15)])
def test_plain_model(cuda_lib, precision, every, skin):
    cfg = configs.ta_config((5, 4, 4), temp=1500.0, jitter=0.05, seed=3)
    compare(configs.snap_params(6, seed=2022), cfg, steps=40, precision=precision, neighevery=every, skin=skin)


def test_two_elements(cuda_lib):
    cfg = configs.ta_config((4, 4, 4), temp=1500.0, jitter=0.05, seed=4)
    types = np.random.default_rng(9).integers(1, 3, cfg.natoms).astype(np.int32)
    compare(configs.snap_params_elements(4, (0.5, 0.45), (1.0, 0.8), chemflag=0, seed=2022), cfg, steps=30, skin=0.03,
            types=types)


def test_surrogate(cuda_lib):
    p8 = configs.snap_params(8, seed=2022)
    cfg = configs.ta_config((5, 5, 5), temp=1500.0, jitter=0.05, seed=5)
    sur = su.Surrogate(configs.snap_params(4, seed=0))
    sur.set_params(su.init_params(3), np.concatenate([np.zeros(14), np.full(14, 1e-3), [-11.7, 0.1]]).astype(np.float32))
    compare(p8, cfg, steps=40, skin=0.04, sur=sur)
    sur.close()
