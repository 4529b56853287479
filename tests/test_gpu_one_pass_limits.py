"""GPU: byte texts of 8 levels at the sizes where they go from one pass to two,
and past them: the limits are read from the code that holds them, and the
launches of a build say which way it went.  Both against passes of 4 levels,
which other tests hold against the oracle."""
import os
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def limit(name):
    with open(os.path.join(ROOT, "pwm_gb300", "csrc", "plain.cu")) as f:
        m = re.search(r"constexpr uint64_t %s = uint64_t\((\d+)\) << (\d+);" % name, f.read())
    return int(m.group(1)) << int(m.group(2))


def built(pg, ctx, d, n, shape):
    """The structures' words, zeros and two levels' blocks, and the build's launches."""
    ds = pg.DeviceStructure(n, 1, 8, matrix=shape[0], tree=shape[1], rank_select=True, context=ctx)
    before = ctx.launches
    ds.build(d.data_ptr())
    launches = ctx.launches - before
    ds.check()
    which = [w for w in (0, 1) if shape[w]]
    got = [ds.download(w) for w in which], [ds.rank_select_blocks(w, l) for w in which for l in (0, 7)]
    ds.free()
    return got, launches


@pytest.mark.parametrize("name,shape", [("kOnePass8Tree", (True, True)), ("kOnePass8Tree", (False, True)),
                                        ("kOnePass8Matrix", (True, False))])
def test_both_sides(pg, name, shape):
    torch = pytest.importorskip("torch")
    most = limit(name)
    ctx, two = pg.Context(), pg.Context()
    two.set_pass_levels(4)
    took = {}
    for n in (most // 2 + 1, most - 1, most, most + 1):
        d = torch.from_numpy(pg.generate(pg.GEN_ZIPF256, n, n, 1)).cuda()
        torch.cuda.synchronize()
        (words, blocks), took[n] = built(pg, ctx, d, n, shape)
        (words2, blocks2), launches2 = built(pg, two, d, n, shape)
        assert (took[n] == launches2) == (n > most), (n, took[n], launches2)
        for a, b in zip(words, words2):
            assert np.array_equal(a.bvs().data, b.bvs().data) and a.zeros() == b.zeros()
        for a, b in zip(blocks, blocks2):
            assert all(np.array_equal(x, y) for x, y in zip(a, b))
    assert took[most - 1] == took[most] != took[most + 1]
