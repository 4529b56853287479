"""GPU: long levels whose rank/select blocks two kernels build (up to 3 levels of
2^22 words and more), against the one kernel that builds the same levels as
part of a deeper structure: every block, sample and count."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGE = 1 << 28  # bits of a level of 2^22 words


def alone(torch, lib, words, nwords):
    """The blocks of one level, by pwmgpu_rank_select_build_noalloc."""
    n12, ns = nwords // 32 + 1, nwords * 64 // 8192 + 2
    t = [torch.full((k,), -1, dtype=d, device="cuda") for k, d in (
        (1, torch.int64), (2 * n12, torch.int32), (ns, torch.int32), (ns, torch.int32), (3, torch.int64))]
    torch.cuda.synchronize()
    p = [ctypes.c_void_p(x.data_ptr()) for x in t]
    assert lib.pwmgpu_rank_select_build_noalloc(ctypes.c_void_p(words), nwords, *p,
                                                ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    l0, l12, s0, s1, counts = (x.cpu().numpy() for x in t)
    return l0.view(np.uint64), l12.view(np.uint32), s0.view(np.uint32)[:counts[0]], s1.view(np.uint32)[:counts[1]]


@pytest.mark.parametrize("n", [EDGE - 64, EDGE, EDGE + 1, EDGE + 2048 * 512 + 1, EDGE + 12345])
def test_against_one_kernel(pg, n):
    torch = pytest.importorskip("torch")
    d = torch.empty(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    pg.generate(pg.GEN_ZIPF256, n, n, 1, device_ptr=d.data_ptr())
    pg.default_context().sync()
    deep = pg.DeviceStructure(n, 1, 8, matrix=True, rank_select=True)
    deep.build(d.data_ptr())
    deep.check()
    v = deep.view(0)
    for level in (0, 5, 7):
        got = alone(torch, pg.default_context().lib, v.words + 8 * v.level_offset[level], (n + 63) // 64)
        assert all(np.array_equal(a, b) for a, b in zip(got, deep.rank_select_blocks(0, level))), level
    # two levels of the matrix and the tree's own, which share the first: 3
    flat = pg.DeviceStructure(n, 1, 2, matrix=True, tree=True, rank_select=True)
    d &= 3
    torch.cuda.synchronize()
    flat.build(d.data_ptr())
    flat.check()
    for which in (0, 1):
        v = flat.view(which)
        for level in (0, 1):
            got = alone(torch, pg.default_context().lib, v.words + 8 * v.level_offset[level], (n + 63) // 64)
            assert all(np.array_equal(a, b) for a, b in zip(got, flat.rank_select_blocks(which, level))), (which, level)
    deep.free()
    flat.free()
