"""Several batches of a process on one device: a short run returns while another thread's long run goes on (beside
it where both grids of resident blocks fit the GPU, between its pieces where they do not), and every trajectory has the bits of a run by itself."""
import threading

import numpy as np
import pytest

import fastmd_b200 as fm
from tests.test_resident_rule_gpu import _chains
from tests.util import run_conf

pytestmark = pytest.mark.gpu
LONG, SHORT = 60_000, 7


def _batch(beads, variant, ens="nvt_langevin 1.0 1.0 1.0 7"):
    b = fm.Batch(max_replicas=1, max_atoms=beads + 4096)
    b.add(run_conf(ensemble=ens, angle=None, nsteps=10_000_000), desc=_chains(beads // 10, 0.3))
    b.set_variants(variant, -1)
    return b


def _read(b):
    x, v, i = b.state(0)
    return [x, v, i, b.thermo(0).as_array()]


# 94 and 938 tiles of 1,184; variant 9 is built for the step graph only
@pytest.mark.parametrize("long, short", [((3000, 0), (3000, 0)), ((30_000, 0), (3000, 0)), ((30_000, 0), (30_000, 0)),
                                         ((30_000, 0), (3000, 9))])
def test_short_run_beside_a_long_one(long, short):
    alone = _batch(*short)
    for n in (SHORT, 120, SHORT):
        alone.run(n)
    want = _read(alone)
    alone.close()
    a, b = _batch(*long), _batch(*short)
    a.run(10)
    started = threading.Event()

    def work():
        started.set()
        a.run(LONG)

    thread = threading.Thread(target=work)
    thread.start()
    started.wait()
    for n in (SHORT, 120, SHORT):
        b.run(n)
    got = _read(b)
    beside = thread.is_alive()
    thread.join()
    assert beside
    assert all(np.array_equal(x, y) for x, y in zip(got, want))
    assert a.info(0).step == LONG + 10 and a.info(0).status_word == 0 and b.info(0).status_word == 0
    a.close()
    b.close()


def test_many_at_once():
    """Eight systems, together more than the GPU holds, in short and long runs; each as it runs alone."""
    sizes = [(3000, 0), (30_000, 0), (600, 0), (12_000, 9), (3000, 0), (30_000, 0), (6000, 0), (3000, 9)]
    runs = [1, 60, 5, 250, 3, 40, 401]

    def advance(b, out, k):
        for n in runs:
            b.run(n)
            b.thermo(0)
        out[k] = _read(b)

    want, got = {}, {}
    for k, s in enumerate(sizes):
        b = _batch(*s)
        advance(b, want, k)
        b.close()
    batches = [_batch(*s) for s in sizes]
    threads = [threading.Thread(target=advance, args=(b, got, k)) for k, b in enumerate(batches)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k, b in enumerate(batches):
        assert b.info(0).status_word == 0
        assert all(np.array_equal(x, y) for x, y in zip(got[k], want[k]))
        b.close()
