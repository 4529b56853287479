"""GPU: leaf histograms of 14 to 16 levels (16-bit counters in shared memory,
flushed before they can overflow): texts of one symbol, of two that share a
word of counters, skewed and even ones, in lengths around a block's chunk and
step, off a 16-byte boundary, and symbols out of range.  Through whole builds
against the oracle (pwm's wx_ps, include/wx_ps.hpp:37-56)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = {1: np.uint8, 2: np.uint16, 4: np.uint32}


@pytest.mark.parametrize("width,L", [(2, 16), (2, 14), (4, 15), (1, 14)])
def test_counts(pg, orc, width, L):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(L)
    top = (1 << min(L, 8 * width)) - 1
    for kind, n, lead in (("one", 1, 0), ("one", 65536, 1), ("one", 12_000_011, 0), ("two", 20_000_003, 1),
                          ("skewed", 65537, 3), ("skewed", 3_000_001, 0), ("even", 32769 * 160, 1)):
        if kind == "one":
            text = np.full(n, top - 1)
        elif kind == "two":
            text = top - 1 + (np.arange(n) % 3 == 0)
        elif kind == "skewed":
            text = np.minimum(rng.geometric(0.3, n) - 1, top)
        else:
            text = rng.integers(0, top + 1, n)
        text = text.astype(DT[width])
        raw = np.zeros((n + 16) * width, np.uint8)
        raw[lead * width:(lead + n) * width] = text.view(np.uint8)
        d = torch.from_numpy(raw).cuda()
        torch.cuda.synchronize()
        ds = pg.DeviceStructure(n, width, L, matrix=True, tree=True)
        try:
            ds.build(d.data_ptr() + lead * width)
            ds.check()
            ref = orc.build(text, L, False, "ps")
            ws = ds.download(0)
            assert ws.zeros() == [int(z) for z in ref.zeros], (kind, n)
            for l in range(L):
                assert np.array_equal(ws.bvs()[l], ref.level(l)), (kind, n, l)
            ref = orc.build(text, L, True, "ps")
            ws = ds.download(1)
            for l in range(L):
                assert np.array_equal(ws.bvs()[l], ref.level(l)), (kind, n, l)
        finally:
            ds.free()


def test_out_of_range(pg):
    torch = pytest.importorskip("torch")
    text = np.zeros(200_001, np.uint16)
    text[-1] = 1 << 14
    d = torch.from_numpy(text.view(np.int16)).cuda()
    torch.cuda.synchronize()
    ds = pg.DeviceStructure(text.size, 2, 14, matrix=True, tree=True)
    with pytest.raises(pg.PwmGpuError):
        ds.build(d.data_ptr())
        ds.check()
    ds.free()
