"""A batch pinned to a list variant steps with that variant's lists: the many-step launch has the ballot form only,
so the row form (1) takes the step graph, and the autotuner keeps a batch of that launch to the ballot form."""
import numpy as np
import pytest

import fastmd_b200 as fm
from tests.test_resident_gpu import ENS, _melt
from tests.util import run_conf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbr_variant", [0, 1, 2])
def test_pinned_list_variant(nbr_variant):
    # no pruned list with this skin: the forces' grouping shows the list itself
    melt, got = _melt(30, 100, seed=4), []
    for graph_steps in (0, -1):
        b = fm.Batch(max_replicas=1, max_atoms=8000, graph_steps=graph_steps)
        b.add(run_conf(ensemble=ENS["npt"], skin=0.1, dt=0.002, nsteps=10_000), desc=melt)
        b.set_variants(0, nbr_variant)
        b.run(100)
        launches = b.launch_counts()["pre"]
        got.append([*b.state(0), b.thermo(0).as_array()])
        assert launches == (0 if graph_steps == 0 and nbr_variant != 1 else 100)
        b.close()
    assert all(np.array_equal(x, y) for x, y in zip(*got))


def test_autotuned_batch_keeps_its_form():
    b = fm.Batch(max_replicas=1, max_atoms=8000)
    b.add(run_conf(nsteps=10_000), desc=_melt(30, 100, seed=4))
    b.autotune(2)
    assert b.variants()[1] != 1 and b.variants()[0] not in (9, 10)
    before = b.launch_counts()["pre"]
    b.run(20)
    assert b.launch_counts()["pre"] == before
    b.close()
