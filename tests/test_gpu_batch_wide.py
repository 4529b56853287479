"""GPU: batches whose longer texts take tiles of 8 vectors a thread in the
tuned plan, next to texts that do not: lengths a symbol around the change and
around such a tile, 1 to 8 levels, with and without trees, against builds with
forced tiles of 4 vectors and the oracle (pwm's wx_ps, include/wx_ps.hpp:
37-56)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILE = 32768


@pytest.mark.parametrize("tree", [False, True])
def test_wide_texts(pg, orc, tree):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(5)
    parts, levels = [], []
    for L in (1, 2, 3, 4, 7, 8):
        edge = TILE if L <= 4 else 16 * TILE  # the last pass's segments: 1 or 16
        for n in (edge - 1, edge, edge + 1, edge + TILE - 1, edge + TILE + 1, 1000):
            top = (1 << L) - 1
            t = np.minimum(rng.geometric(0.2, n) - 1, top) if n % 2 else rng.integers(0, top + 1, n)
            parts.append(t.astype(np.uint8))
            levels.append(L)
    texts = np.concatenate(parts)
    offsets = np.concatenate([[0], np.cumsum([p.size for p in parts])]).astype(np.uint64)
    d = torch.from_numpy(texts).cuda()
    torch.cuda.synchronize()
    got = []
    for vectors in (0, 4):
        b = pg.Batch(offsets, np.array(levels, np.uint32), word_width=1, tree=tree, context=pg.Context())
        if vectors:
            b.set_tile_vectors(vectors)
        for _ in range(2):  # the second replays the graph
            b.build(d.data_ptr())
            b.check()
        got.append([[b.download(i, which) for which in ((0, 1) if tree else (0,))] for i in range(len(levels))])
        b.free()
    for i, (x, y) in enumerate(zip(*got)):
        for which, (u, v) in enumerate(zip(x, y)):
            assert np.array_equal(u.bvs().data, v.bvs().data), (i, which)
            if not which:
                assert u.zeros() == v.zeros()
    for i in (6, 8, 13, 16, 27, 34):
        ref = orc.build(parts[i], levels[i], False, "ps")
        for l in range(levels[i]):
            assert np.array_equal(got[0][i][0].bvs()[l], ref.level(l)), (i, l)
