"""GPU: a structure created by one context and built or queried by another.

pwmgpu_wx_create zeroes a structure's words, and uploads its level descriptors,
on its context's stream.  Here that stream is busy for a tenth of a second, so
that both come long after the call has returned; a build on a second context
has to come after them all the same.  Against the oracle (pwm's wx_ps, include/wx_ps.hpp:37-56).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BUSY_CYCLES = 200_000_000  # about 0.1 s at 2 GHz


def check(ds, orc, text, L):
    for which in (0, 1):
        ref = orc.build(text, L, which == 1, "ps")
        ws = ds.download(which)
        for l in range(L):
            assert np.array_equal(ws.bvs()[l], ref.level(l)), (which, l)


@pytest.mark.parametrize("L,n", [(3, 5001), (8, 70_001), (12, 70_001)])
@pytest.mark.parametrize("rank_select", [False, True])
def test_build_waits_for_the_creation(pg, orc, L, n, rank_select):
    torch = pytest.importorskip("torch")
    busy = torch.cuda.Stream()
    first, second = pg.Context(stream=busy.cuda_stream), pg.Context()
    text = np.random.default_rng(L).integers(0, 1 << L, n).astype(np.uint8 if L <= 8 else np.uint16)
    d = torch.from_numpy(text.view(np.uint8).copy()).cuda()
    torch.cuda.synchronize()
    w = text.itemsize
    warm = pg.DeviceStructure(n, w, L, matrix=True, tree=True, rank_select=rank_select, context=second)
    warm.build(d.data_ptr())  # the second context's scratch
    warm.check()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(BUSY_CYCLES)
    ds = pg.DeviceStructure(n, w, L, matrix=True, tree=True, rank_select=rank_select, context=first)
    ds.ctx = second
    ds.build(d.data_ptr())
    ds.check()
    torch.cuda.synchronize()
    check(ds, orc, text, L)
    if rank_select:
        for which in (0, 1):
            for l in (0, L - 1):
                a, b = ds.rank_select_blocks(which, l), warm.rank_select_blocks(which, l)
                assert all(np.array_equal(x, y) for x, y in zip(a, b))
    ds.free()
    warm.free()
