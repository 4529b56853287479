"""GPU: reduce_alphabet refuses texts and outputs off their symbol's alignment,
before anything is launched (include/pwmgpu.h); an empty text needs none."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PWMGPU_ERR_ARG = 1


@pytest.mark.parametrize("width", [2, 4])
def test_off_the_alignment(pg, width):
    torch = pytest.importorskip("torch")
    n = 1000
    text = np.arange(n * width + 64, dtype=np.uint32).astype(np.uint8)
    d, out = torch.from_numpy(text).cuda(), torch.zeros(n * width + 64, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    for at, to in ((1, 0), (0, 1), (width - 1, 0), (0, width + 1), (1, 1)):
        with pytest.raises(pg.PwmGpuError) as e:
            pg.reduce_alphabet(d.data_ptr() + at, n, width, out.data_ptr() + to)
        assert e.value.status == PWMGPU_ERR_ARG
        assert pg.reduce_alphabet(d.data_ptr() + at, 0, width, out.data_ptr() + to) == (1 << 64) - 1
    torch.cuda.synchronize()
    assert np.array_equal(d.cpu().numpy(), text) and not out.any()
