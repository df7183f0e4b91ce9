"""The launcher's Verlet list at the edges of its two forms (a block per home cell where cells hold four atoms or
more on average, a thread per atom otherwise), of its candidate windows (512) and home groups (64): the list of
every atom, in order, against the candidate order and FP32 predicate restated in numpy (exact)."""
import ctypes as C

import numpy as np
import pytest

import fastmd_b200 as fm

pytestmark = pytest.mark.gpu
F = np.float32


def _expected(xyz, L, rcs, excluded):
    n, nx = len(xyz), max(1, int(F(L) / F(rcs)))
    cell = F(L) / F(nx)
    c = np.floor(xyz * (F(1) / cell)).astype(np.int64) % nx
    cid = (c[:, 2] * nx + c[:, 1]) * nx + c[:, 0]
    order = np.argsort(cid, kind="stable")
    members = [order[cid[order] == k] for k in range(nx ** 3)]
    inv_L, out = F(1) / F(L), []
    for i in range(n):
        cells = []
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    k = ((c[i, 2] + dz) % nx * nx + (c[i, 1] + dy) % nx) * nx + (c[i, 0] + dx) % nx
                    if k not in cells:
                        cells.append(k)
        j = np.concatenate([members[k] for k in cells])
        d = xyz[i] - xyz[j]
        d = d - F(L) * np.rint(d * inv_L)
        r2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]
        j = j[(r2 < F(rcs) * F(rcs)) & (j != i)]
        out.append([int(k) for k in j if int(k) not in excluded[i]])
    return out


@pytest.mark.parametrize("n, L, spill, most_excluded, rows", [
    (107, 9.0, 0.0, 0, 128),     # 27 cells, one atom short of four each: a thread per atom
    (108, 9.0, 0.0, 2, 128),     # four each: a block per cell
    (500, 9.0, 4.0, 3, 512),     # every cell a neighbor; positions outside the box
    (1500, 9.0, 0.0, 40, 1500),  # 1,500 candidates: three windows; more exclusions than lanes
    (2000, 13.0, 0.0, 2, 256),
    (2000, 27.0, 2.0, 0, 256),   # nine cells per axis, two atoms each
    (2100, 24.0, 1.0, 2, 256),   # eight cells per axis, four each: interior cells skip the image
    (1800, 9.0, 0.0, 0, 17),     # overflow: the first rows of each list
])
def test_list_and_order(n, L, spill, most_excluded, rows):
    torch = pytest.importorskip("torch")
    rng, rcs = np.random.default_rng(n), 2.9
    xyz = rng.uniform(-spill, L + spill, (n, 3)).astype(F)
    if n == 1800:
        xyz[:200] = xyz[0] + rng.uniform(0, 0.01, (200, 3)).astype(F)  # over 64 atoms in a cell
    excluded = [set(rng.choice(n, rng.integers(0, most_excluded + 1), replace=False).tolist()) - {i} for i in range(n)]
    expected = _expected(xyz, L, rcs, excluded)
    off = np.concatenate([[0], np.cumsum([len(e) for e in excluded])]).astype(np.int32)
    flat = np.array([j for e in excluded for j in sorted(e)] or [0], np.int32)
    lib, i32 = fm.lib(), dict(dtype=torch.int32, device="cuda")
    pos = torch.from_numpy(np.concatenate([xyz, np.zeros((n, 1), F)], 1)).cuda()
    nbr, cnt, flag = torch.full((rows, n), -1, **i32), torch.zeros(n, **i32), torch.zeros(1, **i32)
    eo, el = torch.from_numpy(off).cuda(), torch.from_numpy(flat).cuda()
    size = C.c_size_t()
    assert lib.fmd_verlet_scratch_bytes(C.c_int32(n), C.c_float(rcs), C.c_float(L), C.byref(size)) == 0
    scratch = torch.empty(size.value, dtype=torch.uint8, device="cuda")

    def p(t):
        return C.c_void_p(t.data_ptr())

    assert lib.fmd_launch_verlet_build(p(pos), C.c_int32(n), C.c_float(L), p(eo) if most_excluded else None,
                                       p(el) if most_excluded else None, C.c_float(rcs), C.c_int32(rows), p(nbr),
                                       p(cnt), p(scratch), size, p(flag), None) == 0
    torch.cuda.synchronize()
    got, counts = nbr.cpu().numpy(), cnt.cpu().numpy()
    assert int(flag.item()) == int(any(len(e) > rows for e in expected))
    for i in range(n):
        assert got[:counts[i], i].tolist() == expected[i][:rows]
