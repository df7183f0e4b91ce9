"""Autotuning and timing the force kernel mid-run leave the state alone: positions, velocities, box and the stored forces that the next step
starts from, tabulated pairs and a barostat included.  Tolerances: the variants group the force sums differently,
1e-5 of forces of order 100; cells of another grid round a position by 5e-7, which a bond's stiffness (below 1,000 per
sigma) turns into 5e-3."""
import ctypes as C

import numpy as np
import pytest

import fastmd_b200 as fm
from tests.test_resident_forms_gpu import _conf, table  # noqa: F401
from tests.test_resident_gpu import _melt

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tabulated", [False, True])
@pytest.mark.parametrize("ens", ["langevin", "nvt", "npt"])
@pytest.mark.parametrize("tune", [True, False])
@pytest.mark.parametrize("graph_steps", [0, -1])
def test_mid_run(table, ens, tabulated, graph_steps, tune):  # noqa: F811
    melt = _melt(20, 50, seed=3, type_block=10)
    b = fm.Batch(max_replicas=2, max_atoms=8000, graph_steps=graph_steps)
    for k in (0, 2):
        b.add(_conf(ens, k, table if tabulated else None), desc=melt)
    b.run(33)
    before = [(*b.state(k), b.last_forces(k), b.info(k).box_L) for k in range(2)]
    if tune:
        b.autotune(2)
    else:
        ms = C.c_double()
        assert fm.lib().fmd_batch_time_force(b._h, C.c_int32(2), C.byref(ms)) == 0 and ms.value > 0
    for k in range(2):
        x0, v0, i0, f0, L = before[k]
        x, v, i = b.state(k)
        assert b.info(k).box_L == L and np.array_equal(v, v0)
        assert np.max(np.abs(x + i * L - x0 - i0 * L)) < 1e-6
        assert np.max(np.abs(b.last_forces(k) - f0)) < 6e-3
    b.run(10)
    assert all(b.info(k).status_word == 0 and b.info(k).step == 43 for k in range(2))
    b.close()
