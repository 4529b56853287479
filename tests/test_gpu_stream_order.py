"""GPU: what a context uploads goes up on its own stream, which alone orders it
before the kernels that read it.

The default stream is kept busy for a tenth of a second.  A copy issued there
would wait for it, and so would the call; a call that uses its context's
stream alone returns with the right answers while the default stream is still
at it.
"""
from contextlib import nullcontext

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BUSY_CYCLES = 200_000_000  # about 0.1 s at 2 GHz


class DefaultStreamBusy:
    """Work on the default stream that must outlast the block."""

    def __enter__(self):
        import torch
        torch.cuda.synchronize()
        torch.cuda._sleep(BUSY_CYCLES)
        self.done = torch.cuda.Event()
        self.done.record()
        return self

    def __exit__(self, kind, value, trace):
        import torch
        waited = self.done.query()
        torch.cuda.synchronize()
        if kind is None:
            assert not waited, "a call waited for the default stream"


def device_words(a):
    import torch
    return torch.from_numpy(np.asarray(a, np.uint64).view(np.int64)).cuda()


@pytest.mark.parametrize("tree", [False, True])
def test_level_descriptors(pg, tree):
    """The rank/select kernels and the queries take their pointers from the
    descriptors that pwmgpu_wx_create uploads."""
    torch = pytest.importorskip("torch")
    n, L, q = 70_001, 8, 500
    rng = np.random.default_rng(5)
    text = rng.integers(0, 256, n).astype(np.uint8)
    ctx = pg.Context()
    d = torch.from_numpy(text).cuda()
    pos = rng.integers(0, n, q)
    d_pos, d_out = device_words(pos), device_words(np.zeros(q))
    kept = []
    for first in (True, False):  # the first time loads the kernels and makes the context's scratch
        with nullcontext() if first else DefaultStreamBusy():
            ds = pg.DeviceStructure(n, 1, L, matrix=not tree, tree=tree, rank_select=True, context=ctx)
            kept.append(ds)  # freeing one would wait for the device
            ds.build(d.data_ptr())
            ds.query(int(tree), pg.Q_ACCESS, d_pos.data_ptr(), None, q, d_out.data_ptr())
            ctx.sync()
    assert np.array_equal(d_out.cpu().numpy(), text[pos].astype(np.int64))
    for ds in kept:
        ds.free()


@pytest.mark.parametrize("width", [1, 2])
def test_huffman_query_tables(pg, width):
    """The code tables that the queries of a Huffman-shaped structure read.  (A
    matrix: the build of a tree frees its source, which waits for the device.)"""
    torch = pytest.importorskip("torch")
    n, q = 70_001, 500
    rng = np.random.default_rng(6)
    text = np.minimum(rng.geometric(0.02, n), 255 if width == 1 else 900).astype(np.uint8 if width == 1 else np.uint16)
    ctx = pg.Context()
    d = torch.from_numpy(text.view(np.uint8).copy()).cuda()
    pos = rng.integers(0, n, q)
    d_pos, d_out = device_words(pos), device_words(np.zeros(q))
    kept = []
    for first in (True, False):
        with nullcontext() if first else DefaultStreamBusy():
            ds = pg.DeviceStructure.huffman(d.data_ptr(), n, width, rank_select=True, context=ctx)
            kept.append(ds)
            ds.query(0, pg.Q_ACCESS, d_pos.data_ptr(), None, q, d_out.data_ptr())
            ctx.sync()
    assert np.array_equal(d_out.cpu().numpy(), text[pos].astype(np.int64))
    for ds in kept:
        ds.free()


@pytest.mark.parametrize("engine", ["tile", "warp"])
def test_batch_plan(pg, orc, engine):
    """The text table, the passes' arguments and the zeroed words of a batch."""
    torch = pytest.importorskip("torch")
    lengths, levels = [1000, 40_003, 0, 70_001], [3, 8, 4, 5]
    offsets = np.concatenate([[0], np.cumsum(lengths)]).astype(np.uint64)
    rng = np.random.default_rng(7)
    texts = [rng.integers(0, 1 << l, n).astype(np.uint8) for n, l in zip(lengths, levels)]
    ctx = pg.Context()
    ctx.set_engine(pg.ENGINE_TILE if engine == "tile" else pg.ENGINE_WARP)
    d = torch.from_numpy(np.concatenate(texts)).cuda()
    kept = []
    for first in (True, False):
        with nullcontext() if first else DefaultStreamBusy():
            b = pg.Batch(offsets, levels, tree=True, context=ctx)
            kept.append(b)
            if engine == "tile":
                b.set_tile_vectors(2)  # no tuning, whose batches are freed
            b.build(d.data_ptr())
            b.check()
    for t, (text, l) in enumerate(zip(texts, levels)):
        for which in (0, 1):
            if text.size:
                ref, ws = orc.build(text, l, which == 1, "ps"), kept[1].download(t, which)
                assert all(np.array_equal(ws.bvs()[m], ref.level(m)) for m in range(l))
    for b in kept:
        b.free()
