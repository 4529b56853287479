"""GPU: tile passes in tiles of 8 or 16 vectors a thread, on both sides of the sizes
where texts take them: texts of one pass, passes that write the next sequence,
last passes over narrowed keys; sizes a symbol around a tile's end, every
symbol width, skewed and even texts, one run a level, texts off a 16-byte
boundary.  Against the oracle (pwm's wx_ps, include/wx_ps.hpp:37-56)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = {1: np.uint8, 2: np.uint16, 4: np.uint32}


@pytest.mark.parametrize("shape", [(True, True), (True, False), (False, True)])
@pytest.mark.parametrize("width,L,edge,tile", [
    (1, 4, 1 << 24, 32768), (1, 3, 1 << 24, 32768), (1, 2, 1 << 24, 32768), (1, 6, 1 << 25, 32768),
    (1, 8, 1 << 25, 32768), (2, 12, 1 << 24, 16384), (2, 11, 1 << 24, 16384), (4, 12, 1 << 23, 8192),
    (4, 9, 1 << 24, 8192), (2, 16, 1 << 21, 16384), (2, 9, 1 << 21, 16384), (4, 20, 1 << 21, 16384),
    (4, 11, 1 << 21, 16384), (4, 18, 1 << 13, 8192)])
def test_sizes_around_the_change(pg, orc, width, L, edge, tile, shape):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(L)
    texts = [("skewed", edge - 1, 0), ("even", edge, width), ("skewed", edge + tile - 1, width),
             ("even", edge + tile + 1, 0), ("single", edge + 65, 0)]
    for kind, n, lead in texts:
        top = (1 << L) - 1
        if kind == "skewed":
            text = np.minimum(rng.geometric(0.02, n) - 1, top).astype(DT[width])
        elif kind == "even":
            text = rng.integers(0, top + 1, n, dtype=DT[width])
        else:
            text = np.full(n, top, DT[width])
        raw = np.zeros(n * width + 16, np.uint8)
        raw[lead:lead + n * width] = text.view(np.uint8)
        d = torch.from_numpy(raw).cuda()
        torch.cuda.synchronize()
        ds = pg.DeviceStructure(n, width, L, matrix=shape[0], tree=shape[1])
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
