"""The plain form's LJ forces with eight, four, two and one lane per atom, at the system sizes where the number
changes, against the FP64 oracle.  Tolerance 1e-12 relative, as for the plain form's other forces: the lanes'
partial sums differ from the oracle's order by rounding only."""
import numpy as np
import pytest

import fastmd_b200 as fm
from oracle import pyoracle as po
from tests.util import oracle_system, rel_rms, run_conf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 18944, 18945, 37889, 75777])
def test_lj_lanes(n):
    rng = np.random.default_rng(n)
    m = int(np.ceil(n ** (1 / 3) - 1e-9))
    L = max(1.1 * m, 9.0)
    k = rng.permutation(m ** 3)[:n]
    xyz = np.stack([k % m, k // m % m, k // (m * m)], 1) * (L / m) + rng.uniform(0.0, 0.1, (n, 3))
    desc = fm.SystemDesc(xyz=xyz, box_L=L, type=np.zeros(n, np.int32), mass=np.ones(1))
    sim = fm.Simulation(run_conf(bond=None, angle=None), desc=desc, form=fm.FMD_FORM_PLAIN_FP64)
    f, pe, vir = sim.forces()
    fo, peo, viro = po.forces(oracle_system(desc, bond=None, angle=None))
    assert rel_rms(f, fo) < 1e-12
    assert abs(pe.sum() - np.sum(peo)) < 1e-12 * abs(np.sum(peo))
    assert np.max(np.abs(vir - viro)) < 1e-11 * np.max(np.abs(viro))
    sim.close()
