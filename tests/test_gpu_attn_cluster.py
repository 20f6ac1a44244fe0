"""Attention by clusters against the three-launch form and the checker: edges of tiles, warps and clusters, windows, head shapes, scores beyond 32 bits (their
base moves), queries beyond int32, probabilities of three bytes; and the other small kernels of a step of several rows."""
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


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("hd", [64, 128])
def test_scores_that_move_the_base_count_as_before(hd, wide):
    """Twelve tiles per CTA, three per warp: scores of the second lie just below the reach of the first one's base, those of the third just
    above it, so that the base moves while the second tile's scores still have weight.  Against the checker."""
    import torch

    from integer_inference_engine_b200 import device
    from oracle import qk_oracle as o
    H, pos, fa = 8, 3071, 16
    rng = np.random.default_rng(hd)
    inv_sqrt = 1 << 13
    q = np.zeros((1, H, hd), np.int64)
    q[0, :, 0] = 1 << 22                                                # score = 8 k[0] + what k[1] adds
    q[0, :, 1] = rng.integers(-(1 << 15), 1 << 15, size=H)
    if wide:
        q[0, 0, 2] = 1 << 33                                            # beyond int32 (over a zero key column): the 64-bit products
    level = (np.arange(pos + 1) // 128) % 3
    k = np.zeros((1, pos + 1, hd), np.int64)
    k[0, :, 0] = np.array([0, (1 << 28) - 3, (1 << 28) + 5])[level] + rng.integers(-2, 3, size=pos + 1)
    k[0, :, 1] = rng.integers(-64, 64, size=pos + 1)
    v = rng.integers(-(1 << 20), 1 << 20, size=(1, pos + 1, hd), dtype=np.int64)
    want = o.attention_cached(q, k, v, pos, H, 1, fa, None, inv_sqrt)
    dev = lambda a, t=torch.int64: torch.from_numpy(np.ascontiguousarray(a)).to("cuda", t)
    device.read_flags()
    got = device.attention_decode_batch(dev(q.reshape(1, -1)), dev(k[:, pos]), dev(v[:, pos]), dev(k.reshape(1, *k.shape), torch.int32), dev(v.reshape(1, *v.shape), torch.int32), pos, H, 1,
                                        hd, fa, inv_sqrt=inv_sqrt)
    assert device.read_flags() == 0
    assert np.array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize(("pos", "H", "Hkv", "hd", "window", "rope", "fa"), [(0, 8, 1, 64, 0, 1, 16), (95, 6, 2, 128, 0, 2, 16), (517, 8, 2, 64, 300, 1, 16),
                                                                            (1025, 4, 1, 128, 0, 0, 22), (640, 16, 2, 64, 641, 2, 12)])
def test_cluster_form_against_the_checker(pos, H, Hkv, hd, window, rope, fa):
    import torch

    from integer_inference_engine_b200 import device
    from integer_inference_engine_b200.model import rope_tables
    from oracle import qk_oracle as o
    B, rng = 3, np.random.default_rng(pos + hd)
    q, k, v = (rng.integers(-(1 << 18), 1 << 18, size=(B, n * hd), dtype=np.int64) for n in (H, Hkv, Hkv))
    kc, vc = (rng.integers(-(1 << 18), 1 << 18, size=(B, Hkv, pos + 2, hd), dtype=np.int64) for _ in range(2))
    cos, sin = (np.ascontiguousarray(t, np.int64) for t in rope_tables(pos + 1, hd, 50000.0, fa))
    dev = lambda a, t=torch.int64: torch.from_numpy(np.ascontiguousarray(a)).to("cuda", t)
    device.read_flags()
    got = device.attention_decode_batch(dev(q), dev(k), dev(v), dev(kc, torch.int32), dev(vc, torch.int32), pos, H, Hkv, hd, fa, window, dev(cos), dev(sin), rope)
    for b in range(B):
        turn = lambda a, n: o.rope_fixed(a.reshape(n, 1, hd), cos[pos:pos + 1], sin[pos:pos + 1], fa, neox=rope == 2) if rope else a.reshape(n, 1, hd)
        kc[b, :, pos], vc[b, :, pos] = turn(k[b], Hkv)[:, 0], v[b].reshape(Hkv, hd)
        want = o.attention_cached(turn(q[b], H).transpose(1, 0, 2), kc[b][:, :pos + 1], vc[b][:, :pos + 1], pos, H, Hkv, fa, window or None)
        assert np.array_equal(got[b:b + 1].cpu().numpy(), want), b
    assert device.read_flags() == 0


def test_column_slices_as_rows():
    import torch

    from integer_inference_engine_b200 import device
    B, H, Hkv, hd, pos = 3, 8, 2, 128, 77
    gen = torch.Generator(device="cuda").manual_seed(3)
    qkv = torch.randint(-(1 << 18), 1 << 18, (B, (H + 2 * Hkv) * hd), generator=gen, device="cuda", dtype=torch.int64)
    kc = torch.randint(-(1 << 18), 1 << 18, (B, Hkv, pos + 1, hd), generator=gen, device="cuda", dtype=torch.int32)
    parts = qkv[:, :H * hd], qkv[:, H * hd:(H + Hkv) * hd], qkv[:, (H + Hkv) * hd:]
    caches = [(kc.clone(), kc.flip(0).contiguous()) for _ in range(2)]
    a = device.attention_decode_batch(*parts, *caches[0], pos, H, Hkv, hd)
    b = device.attention_decode_batch(*(p.contiguous() for p in parts), *caches[1], pos, H, Hkv, hd)
    assert torch.equal(a, b) and all(torch.equal(x, y) for x, y in zip(*caches))


@pytest.mark.parametrize(("rows", "n"), [(1, 32768), (7, 151936), (3, 100001), (32, 32771), (33, 40001), (64, 65536), (65, 33333), (128, 32769), (129, 40000)])
def test_argmax_rows_shared_by_a_cluster(rows, n):
    import torch

    from integer_inference_engine_b200 import device
    x = torch.randint(-50, 50, (rows, n), generator=torch.Generator(device="cuda").manual_seed(n), device="cuda", dtype=torch.int64)
    x[:, n - 1] = 50
    x[0, n // 2] = 50                                                   # ties: the lower index
    assert device.argmax_rows(x).cpu().tolist() == np.argmax(x.cpu().numpy(), axis=1).tolist()


def test_argmax_rows_back_to_back():
    """Clusters of one call start while those of the call before still exchange their candidates."""
    import torch

    from integer_inference_engine_b200 import device
    xs = [torch.randint(-(1 << 40), 1 << 40, (128, 32768), generator=torch.Generator(device="cuda").manual_seed(i), device="cuda") for i in range(4)]
    got = [device.argmax_rows(xs[i % 4]) for i in range(64)]
    want = [np.argmax(x.cpu().numpy(), axis=1) for x in xs]
    assert all(np.array_equal(g.cpu().numpy(), want[i % 4]) for i, g in enumerate(got))


@pytest.mark.parametrize(("experts", "k"), [(5, 5), (128, 8), (300, 40), (1024, 64)])
def test_topk_order_ties_and_gates(experts, k):
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    from oracle import qk_oracle as o
    rng = np.random.default_rng(experts + k)
    rows, d = 9, 256
    h = rng.integers(-(1 << 20), 1 << 20, size=(rows, d), dtype=np.int64)
    router = rng.integers(-(1 << 14), 1 << 14, size=(experts, d), dtype=np.int64)
    router[experts // 2:] = router[:experts - experts // 2]             # equal logits
    handle = qk_cuda.register_i64(router)
    device.read_flags()
    ids, gates = device.route(handle, k, torch.from_numpy(h).cuda(), 16, 24)
    logits = o.linear(h, router, 24)
    want = np.stack([o.topk_lowidx(r, k) for r in logits])
    assert np.array_equal(ids.cpu().numpy(), want)
    assert np.array_equal(gates.cpu().numpy(), np.stack([o.sigmoid_fixed(logits[t][want[t]].astype(np.int64), 16) for t in range(rows)]))
    assert device.read_flags() == 0
    qk_cuda.free_all()
