"""A list buffer that changes the cell grid (cells of rc + buffer), mid-run: the positions and forces of every atom
stay what they are, and the run goes on as one whose buffer was left alone.  Tolerances: a position is an FP32 offset
in a cell below 8 sigma, so two grids' values differ by half an ulp of it each, 5e-7; a force then differs by that
times the stiffness of a bond (below 1,000 per sigma) over a few neighbors, 5e-3; 40 steps of 0.001 let a difference
of 5e-7 grow by less than a hundred."""
import numpy as np
import pytest

import fastmd_b200 as fm
from tests.test_resident_rule_gpu import _chains
from tests.util import run_conf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph_steps", [0, -1])
@pytest.mark.parametrize("ens", ["nvt_langevin 1.0 1.0 1.0 3", "nvt_nh 1.0 1.0 0.5 3", "npt_nh 1.0 1.0 0.5 0.0 0.0 5.0 3"])
@pytest.mark.parametrize("first, then", [(0.1, 0.4), (0.4, 0.1), (0.3, 0.31)])
def test_grid_follows_the_buffer(first, then, ens, graph_steps):
    melt = _chains(120, 0.02)
    melt.vel = np.random.default_rng(5).standard_normal((len(melt.type), 3))
    b, same = (fm.Batch(max_replicas=1, max_atoms=20_000, graph_steps=graph_steps) for _ in range(2))
    for k in (b, same):
        k.add(run_conf(angle=None, skin=first, ensemble=ens, nsteps=10_000), desc=melt)
        k.run(33)
    x0, v0, i0 = b.state(0)
    f0, L = b.last_forces(0), b.info(0).box_L
    b.set_list_buffer(0, then)
    x, v, i = b.state(0)
    assert np.max(np.abs(x + i * L - x0 - i0 * L)) < 1e-6 and np.array_equal(v, v0)
    assert np.max(np.abs(b.last_forces(0) - f0)) < 5e-3
    b.run(40)
    same.run(40)
    assert b.info(0).status_word == 0 and b.info(0).step == 73
    xb, _, ib = b.state(0)
    xs, _, i_s = same.state(0)
    assert np.max(np.abs(xb + ib * b.info(0).box_L - xs - i_s * same.info(0).box_L)) < 5e-5
    b.close()
    same.close()
