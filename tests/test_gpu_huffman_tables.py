"""GPU: Huffman-shaped builds through the key tables in shared memory (8-bit
texts; 16-bit ones from 2^20 symbols on, keys of 16, 17 to 24 and more bits) and
the device's table counts, at text sizes beside the vectors of a thread, texts
off a 16-byte boundary, caller's codes and pwm's, symbols without a code.
Against the oracle (pwm's wx_huff_naive, include/huffman/huff_naive.hpp:
19-126)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(ds, ref, tree, what):
    ws = ds.download(1 if tree else 0)
    assert ws.levels() == ref.levels, what
    assert [ws.bvs().level_bit_size(l) for l in range(ws.levels())] == ref.level_bits, what
    for l in range(ref.levels):
        assert np.array_equal(np.asarray(ws.bvs()[l]), ref.level(l)), (what, l)
    if not tree:
        assert ws.zeros() == [int(z) for z in ref.zeros], what


def build(pg, text, lead, tree, codes=None):
    torch = pytest.importorskip("torch")
    w = text.dtype.itemsize
    raw = np.zeros(text.nbytes + 64, np.uint8)
    raw[lead * w:lead * w + text.nbytes] = text.view(np.uint8)
    d = torch.from_numpy(raw).cuda()
    torch.cuda.synchronize()
    ds = pg.DeviceStructure.huffman(d.data_ptr() + lead * w, text.size, w, tree=tree, codes=codes)
    ds.check()
    return ds


def text16(kind, n):
    rng = np.random.default_rng(n)
    if kind == "short":  # codes of at most 15 bits: 16-bit keys
        return rng.integers(0, 4000, n).astype(np.uint16)
    if kind == "middle":  # 17 to 24 key bits
        return np.where(rng.random(n) < 0.5, rng.integers(0, 65536, n), rng.geometric(0.01, n) % 65536).astype(np.uint16)
    # halving frequencies: codes past 24 bits
    top = int(np.log2(n))
    return np.concatenate([np.full(n >> (k + 1), 257 * k, np.uint16) for k in range(top)] +
                          [np.full(n - sum(n >> (k + 1) for k in range(top)), 9, np.uint16)])


@pytest.mark.parametrize("tree", [False, True])
@pytest.mark.parametrize("kind", ["short", "middle", "long"])
def test_wide_symbols(pg, orc, kind, tree):
    n0 = (1 << 25) + 11 if kind == "long" else (1 << 20) + 5
    for n, lead in ((n0, 0), (n0, 1)) if kind != "long" else ((n0, 0),):
        text = text16(kind, n)
        ref = orc.huff_build(text, tree)
        lo, hi = {"short": (9, 15), "middle": (16, 23), "long": (24, 40)}[kind]
        assert lo <= ref.levels <= hi, ref.levels
        ds = build(pg, text, lead, tree)
        check(ds, ref, tree, (kind, n, lead))
        ds.free()


@pytest.mark.parametrize("tree", [False, True])
@pytest.mark.parametrize("distinct", [5, 200])
def test_bytes(pg, orc, distinct, tree):
    rng = np.random.default_rng(distinct)
    for n in (1, 7, 16, 17, 1023, 1025, 300_001):
        text = np.minimum(rng.geometric(0.02, n), distinct).astype(np.uint8)
        ref = orc.huff_build(text, tree)
        for lead in (0, 3):
            ds = build(pg, text, lead, tree)
            check(ds, ref, tree, (n, lead))
            ds.free()


def test_symbol_without_a_code(pg):
    for dtype, n in ((np.uint8, 5000), (np.uint16, 5000), (np.uint16, (1 << 20) + 9)):
        ln = np.array([1, 2, 2], np.uint64)
        wd = np.array([0, 2, 3], np.uint64)
        text = (np.arange(n) % 3).astype(dtype)
        build(pg, text, 0, False, (ln, wd)).free()
        text[n // 2] = 3
        with pytest.raises(pg.PwmGpuError):
            build(pg, text, 0, False, (ln, wd))
        ln[1] = 0
        text[n // 2] = 0
        with pytest.raises(pg.PwmGpuError):
            build(pg, text, 0, False, (ln, wd))
