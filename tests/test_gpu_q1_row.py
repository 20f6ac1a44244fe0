"""Single-row Q1_0 products at the edges of their launch: odd block counts, parts of a long row, more tiles than ring slots, several
matrices of one width, narrow and wide digits, residuals in and out of place; and one whole decoder layer on shapes around them."""
import numpy as np
import pytest

from oracle import native as onat
from oracle import qk_oracle as o

pytestmark = pytest.mark.gpu
FRAC = 16


@pytest.fixture(autouse=True)
def _weights():
    from integer_inference_engine_b200 import q1_gpu
    yield
    q1_gpu.q1_free_weights()


@pytest.mark.parametrize(("out_f", "nb"), [(1, 1), (17, 31), (2360, 32), (31000, 3), (40, 33), (300, 64), (16 * 148, 65), (70, 131)])
@pytest.mark.parametrize("magnitude", [20, 31, 62])
def test_products(out_f, nb, magnitude):
    import torch

    from integer_inference_engine_b200 import device, q1_gpu
    rng = np.random.default_rng(out_f + 100 * nb + magnitude)
    bits, scale = o.synth_q1(rng, out_f, nb)
    h = q1_gpu.q1_register_weight(bits, scale.astype(np.int32))
    K = nb * 128
    x = rng.integers(-(1 << magnitude), 1 << magnitude, size=(1, K), dtype=np.int64)
    x[0, :3] = [0x7F7F7F7F, -0x80808080, (0x7F7F7F80 if magnitude > 31 else 0)]
    res = rng.integers(-(1 << 40), 1 << 40, size=(1, out_f), dtype=np.int64)
    want = onat.q1_linear(x, bits, scale, FRAC)
    cuda = lambda a: torch.from_numpy(a).cuda()
    out = torch.empty((1, out_f), dtype=torch.int64, device="cuda")
    device.read_flags()
    assert np.array_equal(q1_gpu.apply_fused_dev(h, cuda(x), FRAC, out).cpu().numpy(), want)
    assert np.array_equal(q1_gpu.apply_fused_dev(h, cuda(x), FRAC, out, add=cuda(res)).cpu().numpy(), want + res)
    out.copy_(cuda(res))
    assert np.array_equal(q1_gpu.apply_fused_dev(h, cuda(x), FRAC, out, add=out).cpu().numpy(), want + res)
    over = torch.empty(max(K, out_f) + 1, dtype=torch.int64, device="cuda")          # the row under its own output, misaligned
    over[1:1 + K] = cuda(x[0])
    assert np.array_equal(q1_gpu.apply_fused_dev(h, over[1:1 + K].view(1, K), FRAC, over[:out_f].view(1, out_f)).cpu().numpy(), want)
    if K <= 8192:
        gain = rng.integers(-(1 << 17), 1 << 17, size=K, dtype=np.int64)
        xs = x >> (0 if magnitude < 56 else 8)
        got = q1_gpu.apply_fused_dev(h, cuda(xs), FRAC, out, norm=True, gain=cuda(gain)).cpu().numpy()
        assert np.array_equal(got, onat.q1_linear(o.rmsnorm_fixed(xs, FRAC, 1, gain), bits, scale, FRAC))
    assert device.read_flags() == 0


def test_gain_written_by_the_kernel_in_front():
    """Gain and row come from the kernel launched just before the product, whose start overlaps that kernel's end."""
    import torch

    from integer_inference_engine_b200 import device, q1_gpu
    rng = np.random.default_rng(77)
    K, out_f = 4096, 600
    bits, scale = o.synth_q1(rng, out_f, K // 128)
    h = q1_gpu.q1_register_weight(bits, scale.astype(np.int32))
    xs = rng.integers(-(1 << 20), 1 << 20, size=(8, 1, K), dtype=np.int64)
    gains = rng.integers(-(1 << 17), 1 << 17, size=(8, K), dtype=np.int64)
    xd, gd = torch.from_numpy(xs).cuda(), torch.from_numpy(gains).cuda()
    x, gain = torch.zeros((1, K), dtype=torch.int64, device="cuda"), torch.zeros(K + 1, dtype=torch.int64, device="cuda")[1:]
    device.read_flags()
    outs = []
    for i in range(64):
        x.copy_(xd[i % 8])
        gain.copy_(gd[i % 8])
        outs.append(q1_gpu.apply_fused_dev(h, x, FRAC, torch.empty((1, out_f), dtype=torch.int64, device="cuda"), norm=True, gain=gain))
    want = [onat.q1_linear(o.rmsnorm_fixed(xs[i], FRAC, 1, gains[i]), bits, scale, FRAC) for i in range(8)]
    assert all(np.array_equal(out.cpu().numpy(), want[i % 8]) for i, out in enumerate(outs))
    assert device.read_flags() == 0


@pytest.mark.parametrize(("d", "H", "Hkv", "hd", "ffn", "context"), [(256, 4, 2, 64, 384, 70), (4224, 4, 1, 128, 256, 33), (512, 8, 8, 32, 128, 40),
                                                                     (384, 48, 3, 64, 256, 20)])
def test_decoder_steps(d, H, Hkv, hd, ffn, context):
    """Rows of one and of two parts, head shapes with and without the one-launch attention, against the CPU checker."""
    import torch

    from integer_inference_engine_b200 import device
    from integer_inference_engine_b200.q1_model import SyntheticQ1Decoder
    from oracle import model_oracle
    m = SyntheticQ1Decoder(n_layers=2, d_model=d, n_heads=H, n_kv=Hkv, head_dim=hd, d_ffn=ffn, vocab=300, context=context, max_new=8,
                           seed=d + H, keep_host=True)
    layers = [dict(L, k=L["k"].cpu().numpy().astype(np.int64), v=L["v"].cpu().numpy().astype(np.int64)) for L in m.host_layers]
    cfg = dict(d=m.d, H=m.H, Hkv=m.Hkv, hd=m.hd, ffn=m.ffn, frac=FRAC)
    token, pos = 11, context
    m.token.fill_(token)
    device.read_flags()
    m.capture(context + 4)
    for _ in range(3):
        want, trace, logits = model_oracle.q1_decode_token(token, pos, layers, m.host_top, cfg, m.cos.cpu().numpy(), m.sin.cpu().numpy())
        m.replay()
        torch.cuda.synchronize()
        assert device.read_flags() == 0
        assert np.array_equal(m.x.cpu().numpy(), trace[-1:]) and np.array_equal(m.logits.cpu().numpy()[0], logits)
        assert int(m.token.item()) == want
        token, pos = want, pos + 1
