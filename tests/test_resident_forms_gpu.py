"""The forms of the many-step launch that the sizes, force variants and other replicas choose, each against the
kernels launched one by one (graph_steps = -1), bit for bit: positions staged in shared memory (up to 1,536 beads in
the largest replica) or not, one and two batches per compensated add with four lanes per atom, a group of more than
128 blocks beside another, and the largest system with a block per tile."""
import numpy as np
import pytest

import fastmd_b200 as fm
from tests.test_resident_gpu import ENS, _melt
from tests.util import run_conf

pytestmark = pytest.mark.gpu


def _compare(confs, melts, runs, variant):
    got = []
    for graph_steps in (0, -1):
        b = fm.Batch(max_replicas=len(confs), max_atoms=sum(len(m.type) + 256 for m in melts) + 4096,
                     graph_steps=graph_steps)
        slots = [b.add(c, desc=m) for c, m in zip(confs, melts)]
        b.set_variants(variant, -1)
        out, before = [], b.launch_counts()["pre"]
        for n in runs:
            b.run(n)
            for s in slots:
                row = b.thermo(s)
                out += [*b.state(s), row.as_array(), np.array([row.step, b.info(s).rebuilds, b.info(s).status_word])]
        assert (b.launch_counts()["pre"] == before) == (graph_steps == 0)  # the many-step launch, or not
        b.close()
        got.append(out)
    for a, c in zip(*got):
        assert np.array_equal(a, c)
    assert all(np.all(np.isfinite(a)) for a in got[0])


@pytest.fixture(scope="module")
def table(tmp_path_factory):
    r = np.linspace(0.05, 2.5, 501)
    p = tmp_path_factory.mktemp("table") / "soft.table"
    p.write_text("SOFT\nN 501 R 0.05 2.5\n\n" +
                 "".join(f"{k + 1} {a:.9g} {1 + np.cos(np.pi * a / 2.5):.9g} {np.sin(np.pi * a / 2.5) / a:.9g}\n"
                         for k, a in enumerate(r)))
    return p


def _conf(ens, k, table=None):
    lj = [(0, 0, 1.0, 1.0), (1, 1, 1.0, 1.0)] + ([] if table else [(0, 1, 0.8, 1.0)])
    extra = "thermo 1 5 t.dat\nstress 1 7 s.dat" + (f"\ntable 0 1 {table} SOFT" if table else "")
    return run_conf(ensemble=ENS[ens], ntypes=2, lj=lj, nsteps=29 if k % 5 == 1 else 10_000, extra=extra)


@pytest.mark.parametrize("tabulated", [False, True])
@pytest.mark.parametrize("variant", [0, 1, 4, 5])
@pytest.mark.parametrize("largest", [1536, 1537])  # the last staged size, and the first that is not
@pytest.mark.parametrize("ens", ["langevin", "nvt"])
def test_shared_blocks(table, ens, largest, variant, tabulated):
    # 45 replicas, 1,400 tiles: one lane per atom
    thousand = _melt(20, 50, seed=3, type_block=10)
    melts = [_melt(largest // 3 if largest % 3 == 0 else 1, 3 if largest % 3 == 0 else largest, seed=5, type_block=1),
             _melt(1, 131, seed=6, type_block=4)] + [thousand] * 43
    _compare([_conf(ens, k, table if tabulated else None) for k in range(len(melts))], melts, (11, 30), variant)


@pytest.mark.parametrize("variant", [1, 3, 5])
@pytest.mark.parametrize("ens", ["langevin", "nvt", "npt"])
@pytest.mark.parametrize("chains, length", [(4, 32), (3, 43), (7, 146), (30, 100)])
def test_tiles_two_batches_per_add(chains, length, ens, variant):
    _compare([run_conf(ensemble=ENS[ens], nsteps=10_000)], [_melt(chains, length, seed=chains)], (1, 45), variant)


@pytest.mark.parametrize("variant", [0, 5])
@pytest.mark.parametrize("ens", ["langevin", "nvt", "npt"])
def test_large_groups_side_by_side(ens, variant):
    # 157 blocks each: neither alone in the grid nor few enough to poll every block's word
    _compare([run_conf(ensemble=ENS[ens], nsteps=10_000), run_conf(ensemble=ENS[ens], nsteps=31)],
             [_melt(50, 100, seed=8), _melt(100, 50, seed=9)], (20, 25), variant)


@pytest.mark.parametrize("ens", ["langevin", "nvt"])
def test_largest_system_by_tiles(ens):
    # 37,887 beads: 1,184 tiles, eight on each of 148 SMs
    _compare([run_conf(ensemble=ENS[ens], nsteps=10_000, extra="thermo 1 10 t.dat")], [_melt(12_629, 3, seed=4)],
             (1, 45), 0)
