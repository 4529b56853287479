"""CPU: the shapes of the tile passes (pwm_gb300/csrc/tile_layout.hpp and
host_tables.hpp, checked by tests/host_logic/shapes.cpp): every pass of a plan
has a kernel, and a launch without one is refused.  GPU: texts of 4-byte symbols whose first pass
takes the widest tiles and its prefixes from the histogram kernel, against the
oracle (pwm's wx_ps, include/wx_ps.hpp:37-56)."""
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_shapes(tmp_path):
    exe = str(tmp_path / "shapes")
    src = os.path.join(ROOT, "tests", "host_logic", "shapes.cpp")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-o", exe, src], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("L", [8, 5])
@pytest.mark.parametrize("tree", [False, True])
def test_wide_tiles_from_the_histogram(pg, orc, L, tree):
    torch = pytest.importorskip("torch")
    ctx = pg.Context()
    ctx.set_pass_levels(4)
    rng = np.random.default_rng(L)
    edge = 1 << 21  # 128 tiles of 16384 symbols
    for n, lead in ((edge - 1, 0), (edge, 0), (edge + 3, 4), (edge + 16384 + 4097, 0), (17 * 16384 * 16 + 5, 0)):
        text = np.minimum(rng.geometric(0.04, n) - 1, (1 << L) - 1).astype(np.uint32)
        raw = np.zeros(4 * n + 16, np.uint8)
        raw[lead:lead + 4 * n] = text.view(np.uint8)
        d = torch.from_numpy(raw).cuda()
        torch.cuda.synchronize()
        ds = pg.DeviceStructure(n, 4, L, matrix=not tree, tree=tree, context=ctx)
        ds.build(d.data_ptr() + lead)
        ds.check()
        ref, ws = orc.build(text, L, tree, "ps"), ds.download(int(tree))
        for l in range(L):
            assert np.array_equal(ws.bvs()[l], ref.level(l)), (n, lead, l)
        ds.free()
