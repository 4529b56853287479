"""GPU: rank/select blocks where the one-pass kernel's look-back and samples
can go wrong: levels of one word, of a few L1 blocks, beside the 512 blocks of
a CTA, of many CTAs, dense, sparse and empty of ones, for a matrix, a tree and
both (level 0 shared), against the oracle's bin_rank_popcnt /
bin_select_popcnt (pwm's include/queries/bin_rank_popcnt.hpp:32-86,
bin_select_popcnt.hpp:38-107)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CTA = 512 * 2048  # bits of one CTA's blocks
SIZES = [1, 64, 2047, 2048, 2049, 4096, CTA - 1, CTA, CTA + 1, CTA + 2048, 20 * CTA + 12345]


@pytest.mark.parametrize("kind", ["dense", "sparse", "zeros"])
@pytest.mark.parametrize("shape", [(True, False), (False, True), (True, True)])
def test_blocks(pg, orc, shape, kind):
    rng = np.random.default_rng(3)
    for n in SIZES:
        if kind == "dense":
            text = rng.integers(0, 4, n).astype(np.uint8)
        else:
            text = np.zeros(n, np.uint8)
            if kind == "sparse":
                text[rng.integers(0, n, max(1, n // 9000))] = rng.integers(1, 4, max(1, n // 9000))
        ds = pg.DeviceStructure(n, 1, 2, matrix=shape[0], tree=shape[1], rank_select=True)
        try:
            ds.build_host(text.ctypes.data)
            for which in (0, 1):
                if not shape[which]:
                    continue
                ref = orc.build(text, 2, which == 1, "ps")
                for level in range(2):
                    want = orc.rank_select_blocks(np.ascontiguousarray(ref.level(level)))
                    got = ds.rank_select_blocks(which, level)
                    for w, g in zip(want, got):
                        assert np.array_equal(np.asarray(w).reshape(-1), g), (n, which, level)
        finally:
            ds.free()
