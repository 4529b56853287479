"""GPU: a wait of the rank/select build that runs out.

A CTA of rank_select_kernel counts 2^20 bits of a level and waits for the
counts before them.  As in test_gpu_timeout.py the failure is made on the host:
with the test hook the levels' first CTAs do not run, so that their counts are
never published (a flag that nothing sets).  A text of one level has no
look-back but this one.  The context's spin limit bounds the wait, the check
reports the timeout, the level's number of ones reads all ones (what
pwmgpu_rank_select_build_noalloc's caller, who has no context, looks at), and
the context then builds the same blocks as before.  No GPU fault, trap or hang
is involved.
"""
import ctypes
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PWMGPU_ERR_TIMEOUT = 4


def ones(ds, n):
    """The level's number of ones, by rank(1, n): n is the end of the last block."""
    a, b, out = (np.array([x], dtype=np.uint64) for x in (1, n, 0))
    p = ctypes.POINTER(ctypes.c_uint64)
    st = ds.ctx.lib.pwmgpu_wx_query_host(ds.ctx.h, ds.h, 0, 1, a.ctypes.data_as(p), b.ctypes.data_as(p), 1,
                                         out.ctypes.data_as(p))
    assert st == 0
    return int(out[0])


@pytest.mark.parametrize("ctas", [2, 3, 40])
def test_wait_expires_and_context_recovers(pg, ctas):
    torch = pytest.importorskip("torch")
    ctx = pg.Context()
    lib = ctx.lib
    n = ctas << 20
    text = np.random.default_rng(ctas).integers(0, 2, n).astype(np.uint8)
    d = torch.from_numpy(text).cuda()
    torch.cuda.synchronize()
    ds = pg.DeviceStructure(n, 1, 1, matrix=True, rank_select=True, context=ctx)
    ds.build(d.data_ptr())
    ds.check()
    want = ds.rank_select_blocks(0, 0)
    assert ones(ds, n) == int(text.sum())
    assert lib.pwmgpu_ctx_set_spin_limit(ctx.h, 4096) == 0
    assert lib.pwmgpu_ctx_test_withhold_tile(ctx.h, 1) == 0
    t0 = time.perf_counter()
    ds.build(d.data_ptr())
    assert lib.pwmgpu_wx_check(ctx.h, ds.h) == PWMGPU_ERR_TIMEOUT
    assert time.perf_counter() - t0 < 0.5  # at the context's limit, not the default (more than a second)
    assert ones(ds, n) == 0xFFFFFFFF  # of all ones the queries hold the low half
    assert lib.pwmgpu_ctx_test_withhold_tile(ctx.h, 0) == 0
    assert lib.pwmgpu_ctx_set_spin_limit(ctx.h, 0) == 0
    ds.build(d.data_ptr())
    ds.check()
    assert all(np.array_equal(x, y) for x, y in zip(ds.rank_select_blocks(0, 0), want))
    assert ones(ds, n) == int(text.sum())
    ds.free()
    ctx.close()


def test_longest_level_without_allocation():
    """pwmgpu_rank_select_build_noalloc at its limit, the whole of its state in
    use: every block's count of ones before it, against counts by torch."""
    torch = pytest.importorskip("torch")
    import pwm_gb300 as pg
    lib = pg.default_context().lib
    nwords = 33423360
    blocks = nwords // 32
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    words = torch.randint(0, 1 << 32, (2 * nwords,), device="cuda", generator=g).to(torch.int32)
    pop = torch.tensor([bin(i).count("1") for i in range(256)], dtype=torch.uint8, device="cuda")
    per = torch.empty(blocks, dtype=torch.int64, device="cuda")
    step = blocks // 16
    for i in range(0, blocks, step):
        b = words[64 * i:64 * (i + step)].view(torch.uint8).view(step, 256)
        per[i:i + step] = pop[b.to(torch.int32)].sum(1, dtype=torch.int64)
    l0 = torch.full((nwords // 67108863 + 1,), -1, dtype=torch.int64, device="cuda")
    l12 = torch.full((2 * (blocks + 1),), -1, dtype=torch.int32, device="cuda")
    s0, s1 = (torch.zeros(nwords * 64 // 8192 + 2, dtype=torch.int32, device="cuda") for _ in range(2))
    counts = torch.full((3,), -1, dtype=torch.int64, device="cuda")
    p = [ctypes.c_void_p(t.data_ptr()) for t in (words, l0, l12, s0, s1, counts)]
    torch.cuda.synchronize()
    st = lib.pwmgpu_rank_select_build_noalloc(p[0], nwords, *p[1:], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert st == 0
    torch.cuda.synchronize()
    assert int(counts[2]) == int(per.sum())
    before = torch.cumsum(per, 0) - per
    assert torch.equal(l12[:2 * blocks:2].to(torch.int64) & 0xFFFFFFFF, before)
    assert l12[2 * blocks:].tolist() == [0, 0] and l0.tolist() == [0]
