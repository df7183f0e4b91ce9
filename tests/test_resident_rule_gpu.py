"""Which form a batch's steps take: the many-step launch (no pre-force kernel runs) or the step graph (one per
step), on both sides of the rule, at sizes where the slower form was once taken."""
import numpy as np
import pytest

import fastmd_b200 as fm
from tests.util import run_conf

pytestmark = pytest.mark.gpu


def _chains(nchains, density, length=10):
    """Straight chains along x on a lattice, nowhere near one another."""
    L = (nchains * length / density) ** (1 / 3)
    nx = max(1, int(L / (length + 0.5)))
    ny = int(np.ceil(np.sqrt(nchains / nx)))
    c = np.arange(nchains)
    origin = np.stack([c % nx * (L / nx), c // nx % ny * (L / ny), c // (nx * ny) * (L / ny)], 1)
    xyz = (origin[:, None] + 0.97 * np.arange(length)[None, :, None] * np.array([1.0, 0, 0])).reshape(-1, 3)
    k = np.arange(nchains * length).reshape(nchains, length)
    bonds = np.stack([k[:, :-1].ravel(), k[:, 1:].ravel()], 1).astype(np.int32)
    return fm.SystemDesc(xyz=xyz % L, box_L=L, type=np.zeros(k.size, np.int32), mass=np.ones(1), bonds=bonds,
                         bond_type=np.zeros(len(bonds), np.int32))


def _resident(melts, steps=100, apart=False, skin=0.3, rc=2.5):
    sides = [max(1, int(m.box_L / 2.8)) for m in melts]
    cells = sum((1 << max(0, s - 1).bit_length()) ** 3 for s in sides)  # a capacity of four cells per atom
    atoms = sum(len(m.type) + 256 for m in melts) * max(1, int(rc / 2) ** 2)  # room for longer lists
    b = fm.Batch(max_replicas=len(melts), max_atoms=max(atoms, cells // 4) + 4096)
    slots = [b.add(run_conf(angle=None, nsteps=10_000, skin=skin, rc=rc), desc=m) for m in melts]
    for s in slots if apart else []:
        b.set_rebuild_cadence(s, 0)
    before = b.launch_counts()["pre"]
    b.run(steps)
    ran = b.launch_counts()["pre"] - before
    assert all(b.info(s).status_word == 0 and b.info(s).step == steps for s in slots)
    b.close()
    assert ran in (0, steps)
    return ran == 0


@pytest.mark.parametrize("replicas, chains, density, resident", [
    (1, 300, 0.05, True), (1, 300, 0.005, False),   # 94 tiles; 23 and 287 home cells per tile
    (1, 1200, 0.02, True), (1, 1200, 0.01, False),  # 32 and 64 sort cells per axis
    (64, 100, 0.1, True), (64, 100, 0.02, False),   # blocks that share chunks
])
def test_sparse_boxes(replicas, chains, density, resident):
    assert _resident([_chains(chains, density)] * replicas) == resident


@pytest.mark.parametrize("density, skin, resident", [(0.05, 0.1, True), (0.02, 0.1, False), (0.02, 0.15, True)])
def test_narrow_skins(density, skin, resident):
    # 16 and 32 sort cells per axis; no pruned list with a skin of 0.1
    assert _resident([_chains(300, density)], skin=skin) == resident


# at density 0.3 a list has room for 256 entries with rc 4.5, for 416 with 5.5 and for 768 with 7
@pytest.mark.parametrize("replicas, beads, rc, resident", [
    (1, 18_000, 7.0, True), (1, 30_000, 7.0, False), (64, 1_000, 7.0, False),  # tiles, too many of them, chunks
    (20, 5_000, 4.5, True), (20, 10_000, 4.5, False), (1, 100_000, 5.5, False)])
def test_long_lists(replicas, beads, rc, resident):
    assert _resident([_chains(beads // 10, 0.3)] * replicas, 20, rc=rc) == resident


@pytest.mark.parametrize("replicas, beads, apart, resident", [
    (1, 100_000, False, True), (1, 160_000, False, False),
    (3, 60_000, False, True), (8, 25_000, False, False),
    (20, 10_000, False, True), (45, 7_000, False, False), (45, 7_000, True, True),
    (200, 1_000, False, True), (450, 1_000, False, False), (450, 1_000, True, False),
])
def test_load(replicas, beads, apart, resident):
    assert _resident([_chains(beads // 10, 0.3)] * replicas, 50, apart) == resident
