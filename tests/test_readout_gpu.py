"""State readout at the edges of its pieces (8,192 atoms) and blocks: positions, velocities and image flags come
back in the order given.  Tolerance: a position is an FP32 offset in a cell edge below 8 sigma, so it is off by at
most half an ulp of that, 2.4e-7, and the FP64 additions around it."""
import numpy as np
import pytest

import fastmd_b200 as fm
from tests.util import run_conf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 255, 257, 8191, 8192, 8193, 16385, 32769])
def test_state_reads_back_in_the_order_given(n):
    rng = np.random.default_rng(n)
    m = int(np.ceil(n ** (1 / 3) - 1e-9))
    L = max(1.1 * m, 9.0)
    site = rng.permutation(m ** 3)[:n]
    xyz = np.stack([site % m, site // m % m, site // (m * m)], 1) * (L / m) + rng.uniform(0.0, 0.05, (n, 3))
    vel = rng.standard_normal((n, 3))
    image = rng.integers(-3, 4, (n, 3)).astype(np.int32)
    desc = fm.SystemDesc(xyz=xyz, box_L=L, type=np.zeros(n, np.int32), vel=vel, image=image, mass=np.ones(1))
    sim = fm.Simulation(run_conf(bond=None, angle=None), desc=desc)
    x, v, i = sim.state()
    assert np.max(np.abs(x - xyz)) < 5e-7
    assert np.array_equal(v, vel.astype(np.float32).astype(np.float64))
    assert np.array_equal(i, image)
    sim.close()
