"""GPU: access, rank and select where the query kernels' block arithmetic can
go wrong: texts ending at and beside the 64-bit word, the 512-bit L2 block, the
2048-bit L1 block and the 8192-occurrence sample, dense and sparse symbols (a
sparse bit's samples lie hundreds of L1 blocks apart), single-kind and mixed
batches, plain and Huffman-shaped.  Access and rank against the text, select
against the oracle's query_support (pwm's include/queries/query_support.hpp)
for the plain shapes and against the text for the Huffman-shaped ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 63, 64, 65, 511, 512, 513, 2047, 2048, 2049, 8191, 8192, 8193, 16385, 65536, 300_007]
KINDS = ["dense", "sparse", "runs"]


def make_text(kind, n):
    rng = np.random.default_rng(n)
    if kind == "dense":
        return rng.integers(0, 8, n).astype(np.uint8)
    if kind == "sparse":  # one symbol in thousands differs from the ordinary one
        t = np.full(n, 2, dtype=np.uint8)
        k = max(1, n // 3000)
        t[rng.integers(0, n, k)] = rng.integers(0, 8, k)
        return t
    return np.repeat(rng.integers(0, 8, n // 1500 + 1), 1500)[:n].astype(np.uint8)


def ask(ds, which, op, a, b):
    a = np.ascontiguousarray(a, dtype=np.uint64)
    b = np.ascontiguousarray(b, dtype=np.uint64)
    out = np.zeros(max(a.size, 1), dtype=np.uint64)
    ds.ctx.check(ds.ctx.lib.pwmgpu_wx_query_host(ds.ctx.h, ds.h, which, op, a.ctypes.data, b.ctypes.data, a.size,
                                                 out.ctypes.data))
    return out[:a.size]


def operands(text):
    n = text.size
    rng = np.random.default_rng(1)
    edges = np.array([p + d for p in range(0, n + 1, 512) for d in (-1, 0, 1)], dtype=np.int64)
    pos = np.unique(np.clip(np.concatenate([edges[rng.permutation(edges.size)[:600]], rng.integers(0, n + 1, 400),
                                            [0, n]]), 0, n))
    counts = np.bincount(text, minlength=8)
    sym, occ = [], []
    for s in np.nonzero(counts)[0]:
        k = np.unique(np.clip(np.concatenate([rng.integers(1, counts[s] + 1, 40), [1, counts[s], 8192, 8193, 8194]]), 1,
                              counts[s]))
        sym += [int(s)] * k.size
        occ += [int(x) for x in k]
    return pos, np.array(sym), np.array(occ)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", SIZES)
def test_plain(pg, orc, kind, n):
    text = make_text(kind, n)
    pos, sym, occ = operands(text)
    ds = pg.DeviceStructure(n, 1, 3, matrix=True, tree=True, rank_select=True)
    try:
        ds.build_host(text.ctypes.data)
        before = np.concatenate([np.zeros((1, 8), np.int64), np.cumsum(text[:, None] == np.arange(8), axis=0)])
        at = np.tile(pos, 8)
        of = np.repeat(np.arange(8), pos.size)
        for which, tree in ((0, False), (1, True)):
            inside = pos[pos < n]
            q = orc.query_support(orc.build(text, 3, tree, "ps"))
            select = [q.select(int(s), int(k)) for s, k in zip(sym, occ)]
            assert np.array_equal(ask(ds, which, pg.Q_ACCESS, inside, inside), text[inside])
            assert np.array_equal(ask(ds, which, pg.Q_RANK, of, at), before[at, of])
            assert ask(ds, which, pg.Q_SELECT, sym, occ).tolist() == select
            mixed = ds.query_batch_host(which, np.concatenate([np.full(sym.size, 2), np.full(at.size, 1)]),
                                        np.concatenate([sym, of]), np.concatenate([occ, at]))
            assert np.array_equal(mixed, np.concatenate([np.array(select), before[at, of]]).astype(np.uint64))
    finally:
        ds.free()


@pytest.mark.parametrize("tree", [False, True])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("n", [2048, 16385, 300_007])
def test_huffman(pg, kind, n, tree):
    torch = pytest.importorskip("torch")
    text = make_text(kind, n)
    pos, sym, occ = operands(text)
    d = torch.from_numpy(text).cuda()
    torch.cuda.synchronize()
    ds = pg.DeviceStructure.huffman(d.data_ptr(), n, 1, tree=tree)
    try:
        which = int(tree)
        inside = pos[pos < n]
        assert np.array_equal(ask(ds, which, pg.Q_ACCESS, inside, inside), text[inside])
        for s in np.unique(text):
            where = np.nonzero(text == s)[0]
            before = np.searchsorted(where, pos)
            assert np.array_equal(ask(ds, which, pg.Q_RANK, np.full(pos.size, s), pos), before)
            mine = occ[sym == s]
            # the occurrence a sample is taken at answers with the sample itself, as pwm does
            mine = mine[(mine - 1) % 8192 != 0]
            assert np.array_equal(ask(ds, which, pg.Q_SELECT, np.full(mine.size, s), mine), where[mine - 1])
    finally:
        ds.free()
