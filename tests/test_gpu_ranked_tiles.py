"""GPU: passes that write the next sequence by one sort of 16 digits (1- and
2-byte keys; 4-byte ones in long texts), against the oracle (pwm's wx_ps,
include/wx_ps.hpp:37-56): sizes around a plane word, a thread's row of keys
and a tile, texts off a 16-byte boundary, segments that begin anywhere (the
trees of the later passes), every narrowing of the keys."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = {1: np.uint8, 2: np.uint16, 4: np.uint32}
SIZES = [1, 31, 32, 33, 63, 64, 65, 127, 129, 4095, 8191, 8193, 16383, 16384, 16385, 32769, 100_003]


@pytest.mark.parametrize("shape", [(True, True), (True, False), (False, True)])
@pytest.mark.parametrize("width,L", [(1, 8), (1, 6), (1, 9), (1, 11), (1, 13), (2, 9), (2, 12), (2, 16), (2, 17),
                                     (2, 22), (4, 11), (4, 14), (4, 18)])
def test_levels(pg, orc, width, L, shape):
    torch = pytest.importorskip("torch")
    ctx = pg.Context()
    ctx.set_pass_levels(4)
    rng = np.random.default_rng(L)
    top = (1 << min(L, 8 * width)) - 1
    for n in SIZES:
        for kind in ("skewed", "even"):
            if kind == "skewed":
                text = np.minimum(rng.geometric(0.03, n) - 1, top).astype(DT[width])
            else:
                text = rng.integers(0, top + 1, n, dtype=DT[width])
            lead = width if kind == "even" else 0
            raw = np.zeros(n * width + 16, np.uint8)
            raw[lead:lead + n * width] = text.view(np.uint8)
            d = torch.from_numpy(raw).cuda()
            torch.cuda.synchronize()
            ds = pg.DeviceStructure(n, width, L, matrix=shape[0], tree=shape[1], context=ctx)
            try:
                ds.build(d.data_ptr() + lead)
                ds.check()
                for which in (0, 1):
                    if not shape[which]:
                        continue
                    ref = orc.build(text, L, which == 1, "ps")
                    ws = ds.download(which)
                    for l in range(L):
                        assert np.array_equal(ws.bvs()[l], ref.level(l)), (kind, n, which, l)
            finally:
                ds.free()
