"""GPU: batches of 8-bit texts of 5 to 12 levels (runs counted by planes, the
histogram by columns): lengths around a vector, a tile and a histogram block,
texts off 16-byte boundaries, every forced tile size, symbols out of range.
Against the oracle (pwm's wx_ps, include/wx_ps.hpp:37-56)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vectors", [0, 1, 4])
def test_levels(pg, orc, vectors):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(11)
    parts, levels = [], []
    for L in (5, 6, 7, 8, 9, 11, 12):
        for n in (1, 15, 17, 4095, 4097, 16385, 16 * 4096 + 1, 16 * 16384 + 3):
            top = min((1 << L) - 1, 255)
            t = np.minimum(rng.geometric(0.02, n) - 1, top) if n % 2 else rng.integers(0, top + 1, n)
            parts.append(t.astype(np.uint8))
            levels.append(L)
    texts = np.concatenate(parts)
    offsets = np.concatenate([[0], np.cumsum([p.size for p in parts])]).astype(np.uint64)
    d = torch.from_numpy(texts).cuda()
    torch.cuda.synchronize()
    b = pg.Batch(offsets, np.array(levels, np.uint32), word_width=1, tree=True, context=pg.Context())
    if vectors:
        b.set_tile_vectors(vectors)
    b.build(d.data_ptr())
    b.check()
    for i, (t, L) in enumerate(zip(parts, levels)):
        for which in (0, 1):
            ref = orc.build(t, L, which == 1, "ps")
            ws = b.download(i, which)
            for l in range(L):
                assert np.array_equal(ws.bvs()[l], ref.level(l)), (t.size, L, which, l)
    b.free()


@pytest.mark.parametrize("L", [5, 7])
def test_out_of_range(pg, L):
    torch = pytest.importorskip("torch")
    texts = np.zeros(50_000, np.uint8)
    texts[49_999] = 1 << L
    d = torch.from_numpy(texts).cuda()
    torch.cuda.synchronize()
    b = pg.Batch(np.array([0, 20_000, 50_000], np.uint64), np.array([L, L], np.uint32), word_width=1, tree=False,
                 context=pg.Context())
    with pytest.raises(pg.PwmGpuError):
        b.build(d.data_ptr())
        b.check()
    b.free()
