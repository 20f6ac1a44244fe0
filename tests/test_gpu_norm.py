"""RMSNorm at the edges of its launch forms (a warp or several per row, odd widths, misaligned rows) and of its 32-bit quotients."""
import numpy as np
import pytest

from oracle import qk_oracle as o

pytestmark = pytest.mark.gpu
FRAC = 16


@pytest.mark.parametrize(("rows", "width"), [(9, 4), (17, 100), (8, 128), (3, 132), (25, 256), (2, 260), (1, 127), (2, 4096), (1, 4100), (2, 6148), (1, 8192)])
@pytest.mark.parametrize("spike", [0, 30, 38, 45, 46, 47, 57])
def test_rows_and_magnitudes(rows, width, spike):
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    rng = np.random.default_rng(rows * 1000 + width + spike)
    x = o.to_fixed(rng.standard_normal((rows, width)) * 4, FRAC)
    if spike:
        x[rows // 2] >>= 12                                        # one large value over small ones: quotients near sqrt(width)
        x[rows // 2, width - 1] = -(1 << spike)
        x[0, 0] = (1 << spike) - 1
    gain = np.rint((np.abs(rng.standard_normal(width)) + 0.5) * (1 << FRAC)).astype(np.int64)
    big = gain.copy()
    big[rng.integers(0, width, 3)] = [(1 << 31) - 1, -(1 << 31), 1 << 33]
    buf = torch.empty(rows * width + 1, dtype=torch.int64, device="cuda")
    device.read_flags()
    try:
        for g, off in ((gain, 0), (gain, 1), (big, 0), (None, 0)):
            xd = buf[off:off + rows * width].view(rows, width)
            xd.copy_(torch.from_numpy(x))
            h = -1 if g is None else qk_cuda.register_i64(g)
            got = device.rmsnorm(xd, h, FRAC, 1).cpu().numpy()
            assert np.array_equal(got, o.rmsnorm_fixed(x, FRAC, 1, g)), (off, g is None)
        assert device.read_flags() == 0
        x[rows - 1, 1] = (1 << 57) + 1                             # outside the envelope: flagged
        device.rmsnorm(torch.from_numpy(x).cuda(), -1, FRAC, 1)
        assert device.read_flags() & 2
    finally:
        qk_cuda.free_all()
