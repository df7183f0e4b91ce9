"""A many-step launch whose waits run out: with a limit of no polls every group of more than one block gives its
replica up at its first barrier, with the default it does not.  The given-up replica is reported and stays where it
is (also in the launches already queued), the others finish with the bits of a run without it, and its slot serves
a new replica."""
import numpy as np
import pytest

import fastmd_b200 as fm
from tests.util import run_conf

pytestmark = pytest.mark.gpu
TIMEOUT = 16


def _melt(nchains, length, density, seed):
    gen = dict(nchains=nchains, chain_length=length, density=density, seed=seed)
    d = fm.generate_melt(*gen.values())
    pre = fm.Simulation(run_conf(), gen=dict(pushoff_steps=300, **gen))
    d.xyz, d.vel, d.image = pre.state()
    pre.close()
    return d


def _state(b, slot):
    x, v, i = b.state(slot)
    row = b.thermo(slot)
    return [x, v, i, row.as_array(), np.array([row.step, b.info(slot).rebuilds])]


@pytest.mark.parametrize("polls", [0, 1])
@pytest.mark.parametrize("large", [(30, 100), (60, 100)])  # groups of 94 and 188 blocks
@pytest.mark.parametrize("ens", ["nvt_langevin 1.0 1.0 1.0 7", "nvt_nh 1.0 1.0 0.5 3"])
def test_waits_run_out(ens, large, polls):
    # 30 beads are one tile: a group of one block waits for nobody
    small, melt = _melt(1, 30, 0.1, 2), _melt(*large, 0.85, 3)
    conf = run_conf(ensemble=ens, nsteps=1_000_000, dt=0.0005)

    def batch():
        return fm.Batch(max_replicas=4, max_atoms=20_000)

    b = batch()
    lone = b.add(conf, desc=small)
    b.run(2600)
    alone = _state(b, lone)
    b.close()

    b = batch()
    lost, kept = b.add(conf, desc=melt), b.add(conf, desc=small)
    b.set_wait_limit(polls)
    b.run(2600)
    assert b.info(lost).status_word & TIMEOUT and not b.info(lost).active
    assert b.info(kept).status_word == 0 and b.info(kept).step == 2600
    for a, c in zip(_state(b, kept), alone):
        assert np.array_equal(a, c)
    at = b.info(lost).step
    assert at < 100
    b.set_wait_limit(1 << 22)
    b.run(10)
    assert b.info(lost).step == at and b.info(kept).step == 2610
    # the slot's cell counts and lists serve the next replica
    b.retire(lost)
    again = b.add(conf, desc=melt)
    b.run(40)
    got = _state(b, again)
    assert b.info(again).status_word == 0
    b.close()
    b = batch()
    fresh = b.add(conf, desc=melt)
    b.run(40)
    for a, c in zip(got, _state(b, fresh)):
        assert np.array_equal(a, c)
    b.close()


def test_push_off_reports_it():
    b = fm.Batch(max_replicas=1, max_atoms=8000)
    b.add(run_conf(), gen=dict(nchains=30, chain_length=100, density=0.85, seed=3, pushoff_steps=50))
    b.set_wait_limit(0)
    with pytest.raises(fm.FastMDError, match="device wait"):  # in the push-off, which must finish before the run
        b.run(5)
    b.close()
    with pytest.raises(fm.FastMDError):
        fm.Batch(max_replicas=1, max_atoms=1000).set_wait_limit(-1)
