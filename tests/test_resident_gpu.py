"""Resident steps (many steps in one launch, a group of blocks per replica) against the kernels launched one by
one (graph_steps = -1): the same operations in the same order, so everything read back is the same bits.  The
sizes are the edges of chunks (128 slots), boxes under three cells per axis, one and four lanes per atom (few and
many chunks), replicas that stop at different steps, and every ensemble."""
import numpy as np
import pytest

import fastmd_b200 as fm
from tests.util import run_conf

pytestmark = pytest.mark.gpu
ENS = {"langevin": "nvt_langevin 1.0 1.2 1.0 7", "nvt": "nvt_nh 1.0 1.0 0.5 3", "npt": "npt_nh 1.0 1.0 0.5 0.5 0.5 5.0 3"}


def _melt(nchains, length, seed, type_block=0):
    d = fm.generate_melt(nchains, length, density=0.85, seed=seed, type_block=type_block)
    pre = fm.Simulation(run_conf(ntypes=d.ntypes), gen=dict(nchains=nchains, chain_length=length, density=0.85,
                                                            seed=seed, type_block=type_block, pushoff_steps=300))
    d.xyz, d.vel, d.image = pre.state()
    pre.close()
    return d


def _same(confs, melts, runs, variant=0, gen=None):
    got = []
    for graph_steps in (0, -1):
        b = fm.Batch(max_replicas=len(confs), max_atoms=sum(len(m.type) + 256 for m in melts) + 4096,
                     graph_steps=graph_steps)
        slots = [b.add(c, desc=None if gen else m, gen=gen) for c, m in zip(confs, melts)]
        b.set_variants(variant, -1)
        out = []
        for n in runs:
            b.run(n)
            for s in slots:
                x, v, i = b.state(s)
                row = b.thermo(s)
                out += [x, v, i, row.as_array(), np.array([row.step, row.box_L, b.info(s).rebuilds, b.info(s).status_word])]
        b.close()
        got.append(out)
    for a, c in zip(*got):
        assert np.array_equal(a, c)
    assert all(np.all(np.isfinite(a)) for a in got[0])


@pytest.mark.parametrize("ens", ["langevin", "nvt", "npt"])
@pytest.mark.parametrize("chains, length", [(1, 127), (4, 32), (3, 43), (20, 25), (7, 146), (30, 100)])
def test_one_replica(chains, length, ens):
    _same([run_conf(ensemble=ENS[ens], nsteps=10_000)], [_melt(chains, length, seed=chains)], (1, 7, 45))


@pytest.mark.parametrize("ens", ["langevin", "nvt"])
@pytest.mark.parametrize("variant", [1, 4])
def test_many_chunks_and_uneven_stops(ens, variant):
    # 1,200 chunks in all: one lane per atom, several chunks per block
    small, large = _melt(6, 50, seed=3), _melt(24, 100, seed=4)
    melts = [small] * 20 + [large] * 60
    confs = [run_conf(ensemble=ENS[ens], nsteps=40 if k % 7 == 0 else 10_000) for k in range(len(melts))]
    _same(confs, melts, (25, 30), variant=variant)


@pytest.mark.parametrize("ens", ["langevin", "nvt"])
def test_two_types_with_table_and_stress(tmp_path, ens):
    r = np.linspace(0.05, 2.5, 501)
    p = tmp_path / "soft.table"
    p.write_text("SOFT\nN 501 R 0.05 2.5\n\n" +
                 "".join(f"{k + 1} {a:.9g} {1 + np.cos(np.pi * a / 2.5):.9g} {np.sin(np.pi * a / 2.5) / a:.9g}\n"
                         for k, a in enumerate(r)))
    conf = run_conf(ensemble=ENS[ens], ntypes=2, nsteps=10_000, lj=[(0, 0, 1.0, 1.0), (1, 1, 1.0, 1.0)],
                    extra=f"table 0 1 {p} SOFT\nthermo 1 5 t.dat\nstress 1 3 s.dat")
    _same([conf], [_melt(10, 60, seed=5, type_block=10)], (11, 40))


@pytest.mark.parametrize("ens", ["langevin", "nvt", "npt"])
def test_step_graph(ens):
    # a variant with two lanes per atom is not built in the resident form: the step graph
    _same([run_conf(ensemble=ENS[ens], nsteps=10_000)] * 2, [_melt(12, 50, seed=6), _melt(3, 43, seed=3)], (60, 45),
          variant=9)


def test_push_off():
    melt = fm.generate_melt(10, 50, density=0.85, seed=9)
    _same([run_conf()], [melt], (1, 5),
          gen=dict(nchains=10, chain_length=50, density=0.85, seed=9, pushoff_steps=120))
