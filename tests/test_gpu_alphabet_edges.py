"""GPU: reduce_alphabet (pwm's include/util/alphabet_util.hpp:18-45) where the
device's sweeps can go wrong: symbols that first occur behind the first sweep
of 2^21, at chunk and vector edges and at the very end, texts that hold every
value early, one symbol, texts starting off a 16-byte boundary (in place and
into an output of the same or another alignment), sizes on both sides of the
renumbering's table."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 15, 16, 17, 4095, (1 << 20) - 1, (1 << 20) + 1, (1 << 21) - 1, (1 << 21) + 1, 5_000_011]
DT = {1: np.uint8, 2: np.uint16, 4: np.uint32}


def expect(text):
    syms, first = np.unique(text, return_index=True)
    order = np.argsort(first)
    ids = np.zeros(syms.size, dtype=np.int64)
    ids[order] = np.arange(syms.size)
    return ids[np.searchsorted(syms, text)].astype(text.dtype), syms.size - 1


def make(kind, width, n):
    rng = np.random.default_rng(n * 8 + width)
    top = {1: 256, 2: 65536, 4: 1 << 18}[width]
    if kind == "all_early":
        return rng.integers(0, top, n).astype(DT[width])
    t = np.full(n, 3, dtype=DT[width])
    if kind == "late":  # rare symbols, many of them first seen far into the text, one at the last position
        k = max(1, n // 5000)
        t[np.sort(rng.integers(0, n, k))] = rng.integers(0, top, k)
        t[-1] = top - 1
    return t


@pytest.mark.parametrize("lead", [0, 3])
@pytest.mark.parametrize("kind", ["all_early", "late", "one"])
@pytest.mark.parametrize("width", [1, 2, 4])
def test_edges(pg, width, kind, lead):
    torch = pytest.importorskip("torch")
    for n in SIZES:
        text = make(kind, width, n)
        want, most = expect(text)
        raw = np.zeros((n + 16) * width, np.uint8)
        raw[lead * width:(lead + n) * width] = text.view(np.uint8)
        for out_lead in (lead, lead + 1, None):  # None: in place
            d = torch.from_numpy(raw.copy()).cuda()
            out = d if out_lead is None else torch.full_like(d, 0xAA)
            at = lead if out_lead is None else out_lead
            torch.cuda.synchronize()
            got = pg.reduce_alphabet(d.data_ptr() + lead * width, n, width, out.data_ptr() + at * width)
            assert got == most, (n, out_lead)
            have = out.cpu().numpy()
            assert np.array_equal(have[at * width:(at + n) * width].view(DT[width]), want), (n, out_lead)
            if out_lead is not None:  # nothing written beside the output
                assert (have[:at * width] == 0xAA).all() and (have[(at + n) * width:] == 0xAA).all()
