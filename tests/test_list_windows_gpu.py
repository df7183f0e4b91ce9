"""The launcher's Verlet list by cells at the edges of its candidate windows of 768: three cells per axis, so that
every atom is a candidate of every cell, one atom to either side of one and of two windows, and full lists that span
three and seven, their cells' atoms shared by up to four blocks; against the candidate order and FP32 predicate restated in numpy (exact)."""
import ctypes as C

import numpy as np
import pytest

import fastmd_b200 as fm
from tests.test_list_cells_gpu import F, _expected

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [767, 768, 769, 1536, 1537, 2400, 5184, 5200])  # 192 and 193 atoms per cell: three and four blocks
@pytest.mark.parametrize("dense", [False, True])  # an even box; 300 atoms in one cell (five passes of 64)
def test_windows(n, dense):
    torch = pytest.importorskip("torch")
    rng, L, rcs = np.random.default_rng(n), 9.0, 2.9
    xyz = rng.uniform(0, L, (n, 3)).astype(F)
    if dense:
        xyz[::2][:300] = 1.4 + rng.uniform(0, 0.2, (300, 3)).astype(F)
    expected = _expected(xyz, L, rcs, [set()] * n)
    lib, size, i32 = fm.lib(), C.c_size_t(), dict(dtype=torch.int32, device="cuda")
    assert lib.fmd_verlet_scratch_bytes(C.c_int32(n), C.c_float(rcs), C.c_float(L), C.byref(size)) == 0
    pos = torch.from_numpy(np.concatenate([xyz, np.zeros((n, 1), F)], 1)).cuda()
    nbr, cnt, flag = torch.full((n, n), -1, **i32), torch.zeros(n, **i32), torch.zeros(1, **i32)
    scratch = torch.empty(size.value, dtype=torch.uint8, device="cuda")

    def p(t):
        return C.c_void_p(t.data_ptr())

    assert lib.fmd_launch_verlet_build(p(pos), C.c_int32(n), C.c_float(L), None, None, C.c_float(rcs), C.c_int32(n),
                                       p(nbr), p(cnt), p(scratch), size, p(flag), None) == 0
    torch.cuda.synchronize()
    got, counts = nbr.cpu().numpy(), cnt.cpu().numpy()
    assert int(flag.item()) == 0
    for i in range(n):
        assert got[:counts[i], i].tolist() == expected[i]
