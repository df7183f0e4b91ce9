"""fmd_launch_verlet_build with scratch at every alignment an int array may have, in a buffer of exactly
fmd_verlet_scratch_bytes() bytes: the list of an aligned scratch, and no byte written past the end.  The sizes lie
on both sides of the rule for the list by cells, whose sorted positions are 16-byte words; at 200 atoms the sort's
own storage decides the scratch's size, at 20,000 the positions do."""
import ctypes as C

import numpy as np
import pytest

import fastmd_b200 as fm

pytestmark = pytest.mark.gpu
GUARD = 64


@pytest.mark.parametrize("n, L", [(100, 9.0), (200, 9.0), (20_000, 40.0)])
def test_scratch_alignment(n, L):
    torch = pytest.importorskip("torch")
    rng, rcs, rows = np.random.default_rng(n), 2.9, 128
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform(0, L, (n, 3))
    pos, lib, size = torch.from_numpy(pos).cuda(), fm.lib(), C.c_size_t()
    assert lib.fmd_verlet_scratch_bytes(C.c_int32(n), C.c_float(rcs), C.c_float(L), C.byref(size)) == 0
    lists = []
    for offset in (0, 4, 8, 12, 20):
        i32 = dict(dtype=torch.int32, device="cuda")
        nbr, cnt, flag = torch.full((rows, n), -1, **i32), torch.zeros(n, **i32), torch.zeros(1, **i32)
        scratch = torch.full((offset + size.value + GUARD,), 0x5A, dtype=torch.uint8, device="cuda")

        def p(t, at=0):
            return C.c_void_p(t.data_ptr() + at)

        assert lib.fmd_launch_verlet_build(p(pos), C.c_int32(n), C.c_float(L), None, None, C.c_float(rcs),
                                           C.c_int32(rows), p(nbr), p(cnt), p(scratch, offset), size, p(flag),
                                           None) == 0
        torch.cuda.synchronize()
        assert bool((scratch[offset + size.value:] == 0x5A).all()) and bool((scratch[:offset] == 0x5A).all())
        lists.append((nbr.cpu().numpy(), cnt.cpu().numpy(), int(flag.item())))
    for nbr, cnt, flag in lists[1:]:
        assert np.array_equal(cnt, lists[0][1]) and np.array_equal(nbr, lists[0][0]) and flag == 0
    assert lists[0][1].sum() > n
