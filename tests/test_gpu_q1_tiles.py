"""Q1_0 products of several tokens on the tensor-core tiles against the CPU oracle, where the tiles can go wrong: token counts
around the tile widths, rows around 128, few and many blocks, one to eight digit planes, scales beyond the three-plane
read-out, shared tiles (added atomically, in place or over cleared outputs) and whole ones."""
import numpy as np
import pytest

from oracle import native as onat
from oracle import qk_oracle as o

pytestmark = pytest.mark.gpu
FRAC = 16


@pytest.mark.parametrize("out_f,nb,T,magbits,scale_bits", [
    (1, 1, 2, 20, 12), (127, 9, 16, 22, 12), (129, 8, 17, 22, 12), (640, 33, 32, 22, 14), (300, 7, 33, 30, 12), (4096, 3, 64, 22, 12),
    (200, 130, 65, 38, 12), (384, 16, 130, 47, 20), (150, 5, 19, 62, 40), (96, 12, 6, 22, 31), (2400, 1, 2047, 22, 12), (130, 4, 8, 22, 12), (257, 9, 2, 62, 40), (64, 35, 7, 30, 12)])
def test_tiles_match_the_oracle(out_f, nb, T, magbits, scale_bits):
    import torch

    from integer_inference_engine_b200 import device, q1_gpu
    rng = np.random.default_rng(out_f * 7 + nb * 3 + T)
    bits, scale = o.synth_q1(rng, out_f, nb)
    lim = 1 << scale_bits
    scale = rng.integers(-lim, lim, size=scale.shape, dtype=np.int64)
    x = rng.integers(-(1 << magbits), 1 << magbits, size=(T, nb * 128), dtype=np.int64)
    if magbits == 22:
        x[0, :3] = [8355711, -8421504, 8355711]                      # the ends of three balanced digits
    device.read_flags()
    h = q1_gpu.q1_register_weight(bits, scale.astype(np.int32) if scale_bits < 31 else scale)
    want = onat.q1_linear(x, bits, scale, FRAC)
    xd = torch.from_numpy(x).cuda()
    assert np.array_equal(q1_gpu.apply_dev(h, xd, FRAC).cpu().numpy(), want)
    other = rng.integers(-(1 << 40), 1 << 40, size=want.shape, dtype=np.int64)
    res = torch.from_numpy(other).cuda()
    q1_gpu.apply_fused_dev(h, xd, FRAC, res, add=res)                 # the residual row in place
    assert np.array_equal(res.cpu().numpy(), want + other)
    out = torch.full(want.shape, 7, dtype=torch.int64, device="cuda")
    q1_gpu.apply_fused_dev(h, xd, FRAC, out, add=torch.from_numpy(other).cuda())
    assert np.array_equal(out.cpu().numpy(), want + other)
    if out_f * T <= xd.numel():                                      # the output over the input
        q1_gpu.apply_dev(h, xd, FRAC, out=xd.view(-1)[:out_f * T].view(T, out_f))
        assert np.array_equal(xd.view(-1)[:out_f * T].view(T, out_f).cpu().numpy(), want)
    assert device.read_flags() == 0


@pytest.mark.parametrize(("nb", "scale"), [(4, (1 << 31) - 1), (4, 2130706431), (4, 2130706432), (2, (1 << 32) - 1), (5, 1717986918), (1, (1 << 32) - 1)])
@pytest.mark.parametrize("T", [2, 16, 70])
def test_largest_sums_of_three_planes(nb, scale, T):
    """Every value at an end of three balanced digits, every sign the same, scales around the point (2^33 - 2^26 over the blocks) where
    the products of a tile still fit 64 bits without a shift in between."""
    import torch

    from integer_inference_engine_b200 import device, q1_gpu
    out_f = 40
    bits = np.zeros((out_f, nb, 16), np.uint8)
    bits[::2] = 0xFF
    scales = np.full((out_f, nb), scale, np.int64)
    scales[::4] *= -1
    x = np.full((T, nb * 128), -8421504, np.int64)
    x[1] = 8355711
    h = q1_gpu.q1_register_weight(bits, scales.astype(np.int32) if scale < 1 << 31 else scales)
    device.read_flags()
    assert np.array_equal(q1_gpu.apply_dev(h, torch.from_numpy(x).cuda(), FRAC).cpu().numpy(), onat.q1_linear(x, bits, scales, FRAC))
    assert device.read_flags() == 0


@pytest.mark.parametrize("T", [1, 2, 9])
def test_rows_that_start_on_eight_bytes(T):
    """Activations, gain, gate and up at odd element offsets and an odd row distance."""
    import torch

    from integer_inference_engine_b200 import device, q1_gpu
    rng = np.random.default_rng(T)
    out_f, nb = 70, 3
    K = nb * 128
    bits, scale = o.synth_q1(rng, out_f, nb)
    h = q1_gpu.q1_register_weight(bits, scale.astype(np.int32))
    odd = lambda a: torch.cat([torch.zeros(1, dtype=torch.int64), torch.from_numpy(a.reshape(-1))]).cuda()[1:].view(a.shape)
    x, gain = rng.integers(-(1 << 20), 1 << 20, size=(T, K), dtype=np.int64), rng.integers(-(1 << 17), 1 << 17, size=K, dtype=np.int64)
    gu = rng.integers(-(1 << 18), 1 << 18, size=(T, 2 * K + 1), dtype=np.int64)
    new = lambda: torch.empty((T, out_f), dtype=torch.int64, device="cuda")
    device.read_flags()
    assert np.array_equal(q1_gpu.apply_dev(h, odd(x), FRAC).cpu().numpy(), onat.q1_linear(x, bits, scale, FRAC))
    got = q1_gpu.apply_fused_dev(h, odd(x), FRAC, new(), norm=True, gain=odd(gain)).cpu().numpy()
    assert np.array_equal(got, onat.q1_linear(o.rmsnorm_fixed(x, FRAC, 1, gain), bits, scale, FRAC))
    g, u = gu[:, :K], gu[:, K + 1:]
    act = ((g * o.sigmoid_fixed(g, FRAC) >> FRAC) * u) >> FRAC
    gud = odd(gu)
    for gd, ud in ((gud[:, :K], gud[:, K + 1:]), (torch.from_numpy(gu).cuda()[:, :K], torch.from_numpy(gu).cuda()[:, K + 1:])):
        got = q1_gpu.apply_fused_dev(h, gd, FRAC, new(), up=ud).cpu().numpy()
        assert np.array_equal(got, onat.q1_linear(act, bits, scale, FRAC))
    assert device.read_flags() == 0
