"""GPU: texts whose levels all come from one tile pass, with every table made
on the device: sizes at the edges of words, of the half-size and the whole
tiles, of the size where the tiles double and where 8 levels go to two passes,
2 to 8 levels, every shape, texts off a 16-byte boundary, host texts, and
symbols out of range.  Against the oracle (pwm's wx_ps, include/wx_ps.hpp:
37-56)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DT = {1: np.uint8, 2: np.uint16, 4: np.uint32}
SIZES = [1, 63, 64, 65, 8191, 8192, 8193, 16385, 150_001, (1 << 21) - 1, (1 << 21) + 1]


def check(ds, orc, text, L):
    for which, tree in ((0, False), (1, True)):
        if not (ds.tree if tree else ds.matrix):
            continue
        ref = orc.build(text, L, tree, "ps")
        ws = ds.download(which)
        for l in range(L):
            assert np.array_equal(ws.bvs()[l], ref.level(l)), (text.size, L, which, l)
        if not tree:
            assert ws.zeros() == [int(z) for z in ref.zeros]


@pytest.mark.parametrize("shape", [(True, False), (False, True), (True, True)])
@pytest.mark.parametrize("width,L", [(1, 8), (1, 7), (1, 5), (1, 4), (1, 2), (2, 7), (2, 3), (4, 6), (4, 2)])
def test_levels(pg, orc, width, L, shape):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(L)
    for n in SIZES:
        text = np.minimum(rng.geometric(0.05, n) - 1, (1 << L) - 1).astype(DT[width])
        raw = np.zeros(n * width + 16, np.uint8)
        raw[width:width * (n + 1)] = text.view(np.uint8)
        for lead, buf in ((0, text.view(np.uint8).copy()), (width, raw)):
            d = torch.from_numpy(buf).cuda()
            torch.cuda.synchronize()
            ds = pg.DeviceStructure(n, width, L, matrix=shape[0], tree=shape[1])
            try:
                ds.build(d.data_ptr() + lead)
                ds.check()
                check(ds, orc, text, L)
            finally:
                ds.free()


@pytest.mark.parametrize("limit,shape", [(30 << 20, (True, True)), (60 << 20, (True, False))])
def test_one_and_two_passes_agree(pg, limit, shape):
    """8 levels on both sides of the limit, against passes of 4 levels."""
    torch = pytest.importorskip("torch")
    ctx = pg.Context()
    two = pg.Context()
    two.set_pass_levels(4)
    which = [w for w in (0, 1) if shape[w]]
    for n in (limit, limit + 1):
        text = pg.generate(pg.GEN_ZIPF256, n, n, 1)
        d = torch.from_numpy(text).cuda()
        torch.cuda.synchronize()
        got = []
        for c in (ctx, two):
            ds = pg.DeviceStructure(n, 1, 8, matrix=shape[0], tree=shape[1], rank_select=True, context=c)
            ds.build(d.data_ptr())
            ds.check()
            got.append(([ds.download(w) for w in which], [ds.rank_select_blocks(w, l) for w in which for l in (0, 7)]))
            ds.free()
        for a, b in zip(got[0][0], got[1][0]):
            assert np.array_equal(a.bvs().data, b.bvs().data) and a.zeros() == b.zeros()
        for a, b in zip(got[0][1], got[1][1]):
            assert all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("tree", [False, True])
@pytest.mark.parametrize("n", [1, 5000, 100_003])
def test_host_texts(pg, orc, n, tree):
    torch = pytest.importorskip("torch")
    text = pg.generate(pg.GEN_ZIPF256, 3, n, 1)
    ref = orc.build(text, 8, tree, "ps")
    ws = pg.wx_ps(np.uint8, tree).compute(text, n, 8)
    pinned = torch.from_numpy(text).pin_memory()
    ds = pg.DeviceStructure(n, 1, 8, matrix=not tree, tree=tree)
    ds.build_host(pinned.data_ptr())
    ds.check()
    pinned.zero_()  # the call has read it
    down = ds.download(int(tree))
    for l in range(8):
        assert np.array_equal(ws.bvs()[l], ref.level(l)) and np.array_equal(down.bvs()[l], ref.level(l))
    ds.free()


def test_symbol_out_of_range(pg, orc):
    torch = pytest.importorskip("torch")
    text = np.arange(20_000, dtype=np.uint32).astype(np.uint8) % 32
    for bad in (0, 9999, 19_999):
        t = text.copy()
        t[bad] = 32
        d = torch.from_numpy(t).cuda()
        torch.cuda.synchronize()
        ds = pg.DeviceStructure(t.size, 1, 5, matrix=True, tree=True, rank_select=True)
        with pytest.raises(pg.PwmGpuError):
            ds.build(d.data_ptr())
        d.copy_(torch.from_numpy(text))
        torch.cuda.synchronize()
        ds.build(d.data_ptr())  # the context is usable
        ds.check()
        check(ds, orc, text, 5)
        ds.free()
