"""Attention by clusters against the three-launch form: edges of tiles, warps and clusters, windows, head shapes, scores beyond 32 bits (their
base moves), queries beyond int32, probabilities of three bytes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(("pos", "H", "Hkv", "hd", "window", "rope", "bits", "fa"), [
    (0, 8, 2, 64, 0, 1, 18, 16), (30, 8, 1, 128, 0, 2, 18, 16), (31, 6, 2, 128, 0, 0, 18, 16), (32, 4, 4, 64, 0, 2, 24, 16), (127, 16, 2, 128, 0, 1, 18, 16),
    (128, 8, 8, 128, 0, 2, 18, 16), (200, 8, 2, 128, 65, 1, 18, 16), (517, 32, 4, 128, 0, 0, 25, 16), (700, 8, 1, 64, 0, 1, 25, 12), (333, 8, 2, 128, 0, 1, 40, 16),
    (150, 4, 1, 128, 0, 2, 20, 22), (1023, 16, 2, 128, 0, 1, 18, 16), (1024, 8, 1, 128, 0, 1, 18, 16), (0, 8, 2, 64, 3, 1, 30, 16), (1, 4, 2, 128, 0, 1, 44, 16),
    (2050, 8, 1, 64, 2000, 1, 18, 16)])
@pytest.mark.parametrize("batch", [1, 5])
def test_cluster_form_gives_the_same_bytes(pos, H, Hkv, hd, window, rope, bits, fa, batch):
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    from integer_inference_engine_b200.model import rope_tables
    gen = torch.Generator(device="cuda").manual_seed(pos * 31 + H + bits + batch)
    r = lambda n, *shape: torch.randint(-(1 << n), 1 << n, shape, generator=gen, device="cuda", dtype=torch.int64)
    kv_bits = min(bits, 30)
    q, k, v = r(bits, batch, H * hd), r(kv_bits, batch, Hkv * hd), r(20, batch, Hkv * hd)
    # a ramp in the keys: later tiles score far above earlier ones
    kc = (r(kv_bits, batch, Hkv, pos + 9, hd) * torch.linspace(0.05, 1, pos + 9, device="cuda").view(1, 1, -1, 1)).to(torch.int32)
    vc = r(30, batch, Hkv, pos + 9, hd).to(torch.int32)
    if bits == 25:
        kc[:, :, pos // 2:pos // 2 + 3] = kc[:, :, pos // 2:pos // 2 + 3].abs()
        q = q.abs()
    cos, sin = (torch.from_numpy(t).cuda() for t in rope_tables(pos + 9, hd, 50000.0, fa))
    lib = qk_cuda._lib()
    results = []
    device.read_flags()
    for form in (0, 1):
        lib.iie_set_attn_fused(form)
        try:
            k1, v1 = kc.clone(), vc.clone()
            out = device.attention_decode_batch(q, k, v, k1, v1, pos, H, Hkv, hd, fa, window, cos, sin, rope)
            results.append([t.cpu().numpy() for t in (out, k1, v1)])
        finally:
            lib.iie_set_attn_fused(1)
    flags = device.read_flags()
    assert flags & ~4 == 0                                             # (a rotated key of 2^30 and more may not fit the cache)
    for a, b in zip(*results):
        assert np.array_equal(a, b)
