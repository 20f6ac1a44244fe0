"""Host-array entries through page-locked staging: sizes on both sides of the staging buffers, activations beyond the digits (the call repeats
with the exact kernel and leaves no flag behind), results that outlive later calls."""
import numpy as np
import pytest

from oracle import native as onat
from oracle import qk_oracle as o

pytestmark = pytest.mark.gpu
FW = 24


@pytest.mark.parametrize("rows", [1, 2, 33, 600])
def test_grouped_products(rows):
    from integer_inference_engine_b200 import device, qk_cuda
    rng = np.random.default_rng(rows)
    nb, widths = 1, (512, 256, 1024)
    raw = [o.synth_q4k(np.random.default_rng(i), w, nb) for i, w in enumerate(widths)]
    hs = [qk_cuda.register_weight(r, w, nb, o.Q4_K) for r, w in zip(raw, widths)]
    device.read_flags()
    kept = []
    for bits in (20, 62, 20):
        x = rng.integers(-(1 << bits), 1 << bits, size=(rows, nb * 256), dtype=np.int64)
        if bits == 62:
            x[:, 1:] >>= 40
            x[-1, 0] = np.iinfo(np.int64).max                          # beyond eight balanced digits
        got = qk_cuda.apply_resident_grouped(hs, x, widths, FW)
        want = [onat.qk_linear(r, x, w, nb, FW, o.Q4_K) for r, w in zip(raw, widths)]
        kept.append((got, want))
        assert device.read_flags() == 0
    for got, want in kept:
        for a, b in zip(got, want):
            assert np.array_equal(a, b)
    qk_cuda.free_all()


@pytest.mark.parametrize("qtype", [o.Q4_K, o.Q6_K])
@pytest.mark.parametrize("nb,widths,bits", [(1, (8, 1), 20), (3, (129, 7, 640), 30), (8, (33, 264, 16, 9), 40), (5, (2000, 3000), 62), (2, (100, 5, 77, 16, 40), 20)])
def test_one_row_with_several_matrices(qtype, nb, widths, bits):
    """Matrices that end in odd half-tiles, one behind the other in one launch (up to four; five take a launch each)."""
    from integer_inference_engine_b200 import device, qk_cuda
    rng = np.random.default_rng(nb)
    synth = o.synth_q4k if qtype == o.Q4_K else o.synth_q6k
    raw = [synth(np.random.default_rng(i + nb), w, nb) for i, w in enumerate(widths)]
    hs = [qk_cuda.register_weight(r, w, nb, qtype) for r, w in zip(raw, widths)]
    device.read_flags()
    x = rng.integers(-(1 << bits), 1 << bits, size=(1, nb * 256), dtype=np.int64)
    got = qk_cuda.apply_resident_grouped(hs, x, widths, FW)
    assert device.read_flags() == 0
    for a, r, w in zip(got, raw, widths):
        assert np.array_equal(a, onat.qk_linear(r, x, w, nb, FW, qtype))
    qk_cuda.free_all()


@pytest.mark.parametrize("formats,beyond,launches", [((o.Q4_K,) * 3, False, 2), ((o.Q6_K,) * 2, False, 2), ((o.Q4_K, o.Q6_K), False, 3), ((o.Q4_K,) * 5, False, 6),
                                                      ((o.Q4_K,) * 3, True, 5), ((o.Q6_K,) * 4, True, 6), ((o.Q6_K, o.Q4_K), True, 5)])
def test_launches_of_one_row_with_several_matrices(formats, beyond, launches):
    """The digits and one launch for up to four matrices of one format, else a launch per matrix; a row beyond eight digits once more through the
    exact kernel, matrix by matrix."""
    from integer_inference_engine_b200 import device, qk_cuda
    nb, widths = 3, (300, 40, 129, 8, 77)[:len(formats)]
    raw = [(o.synth_q4k if q == o.Q4_K else o.synth_q6k)(np.random.default_rng(i), w, nb) for i, (q, w) in enumerate(zip(formats, widths))]
    hs = [qk_cuda.register_weight(r, w, nb, q) for r, w, q in zip(raw, widths, formats)]
    x = np.random.default_rng(9).integers(-(1 << 20), 1 << 20, size=(1, nb * 256), dtype=np.int64)
    if beyond:
        x[0, 300] = np.iinfo(np.int64).max
    device.read_flags()
    before = device.launch_count()
    got = qk_cuda.apply_resident_grouped(hs, x, widths, FW)
    assert device.launch_count() - before == launches
    assert device.read_flags() == 0
    for a, r, w, q in zip(got, raw, widths, formats):
        assert np.array_equal(a, onat.qk_linear(r, x, w, nb, FW, q))
    qk_cuda.free_all()


def test_results_share_no_memory():
    import gc

    from integer_inference_engine_b200 import q1_gpu
    a, b = q1_gpu._result((3, 1 << 16)), q1_gpu._result((1 << 18,))
    a[:], b[:] = 1, 2
    view = a[1]
    del a
    gc.collect()
    c = q1_gpu._result((3, 1 << 16))                                    # the view still holds the first array's memory
    c[:] = 3
    assert (view == 1).all() and (b == 2).all()
    p = c.ctypes.data
    del c
    gc.collect()
    assert q1_gpu._result((3, 1 << 16)).ctypes.data == p                # given back and taken again
    many = [q1_gpu._result((1 << 20,)) for _ in range(12)]              # beyond the pool: ordinary memory
    for i, m in enumerate(many):
        m[:] = i
    assert all((m == i).all() for i, m in enumerate(many))


def _raise_time_out_bit(lib):
    getattr(lib, "_ZN3iie17restore_flag_bitsEi")(8)                     # from the host: what a kernel whose wait gave up leaves


def test_a_wait_that_gave_up_fails_the_call():
    """Bit 3 of the flag word says that outputs were left out: no host-array entry reports success with it."""
    from integer_inference_engine_b200 import device, q1_gpu, qk_cuda
    rng = np.random.default_rng(5)
    d, eff, w = 256, 256, 512
    raw = o.synth_q4k(rng, w, 1)
    h = qk_cuda.register_weight(raw, w, 1, o.Q4_K)
    gate, up = (qk_cuda.register_weight(o.synth_q4k(rng, eff, 1), eff, 1, o.Q4_K) for _ in range(2))
    down = qk_cuda.register_weight(o.synth_q6k(rng, d, 1), d, 1, o.Q6_K)
    bits, scale = o.synth_q1(rng, 64, 2)
    q1 = q1_gpu.q1_register_weight(bits, scale.astype(np.int32))
    x = rng.integers(-(1 << 20), 1 << 20, size=(3, d), dtype=np.int64)
    wide = x.copy()
    wide[0, 0] = np.iinfo(np.int64).max                                 # repeats with the exact kernel
    gates = np.full((3, 1), 1 << 16, np.int64)
    calls = [lambda: qk_cuda.apply_resident(h, x, w, FW), lambda: qk_cuda.apply_resident(h, wide, w, FW),
             lambda: qk_cuda.apply_resident_grouped((h, gate), x, (w, eff), FW), lambda: qk_cuda.apply_resident_grouped((h, gate), wide, (w, eff), FW),
             lambda: qk_cuda.apply_resident_grouped((h, gate), x[:1], (w, eff), FW),
             lambda: qk_cuda.moe_ffn_batched([gate] * 3, [up] * 3, [down] * 3, 3, 1, x, gates, d, eff, 16, FW),
             lambda: q1_gpu.q1_apply_resident(q1, x, 64, 2, 16), lambda: q1_gpu.q1_apply_resident(q1, x[:1], 64, 2, 16),
             lambda: q1_gpu.q1_apply_gpu(x, bits, scale, 16), lambda: q1_gpu.q1_apply_dp4a_gpu(x, bits, scale, 16)]
    device.read_flags()
    for i, call in enumerate(calls):
        good = call()
        assert good is not None, i
        _raise_time_out_bit(qk_cuda.load_library())
        assert call() is None, i
        again = call()                                                  # the bit went with the call that reported it
        for a, b in zip(good, again):
            assert np.array_equal(a, b), i
        assert device.read_flags() == 0, i
    qk_cuda.free_all()
    q1_gpu.q1_free_weights()


@pytest.mark.parametrize("T", [16, 77, 620])
def test_prompt_rows_arrive_whole(T):
    """Rows below, inside and beyond the page-locked buffer they travel through (1 MB, 32 MB): the exported values of every row against the
    checker's product of the normalised row."""
    from integer_inference_engine_b200 import q1_gpu
    rng = np.random.default_rng(T)
    d, H, Hkv, hd, dff, vocab = 8192, 2, 1, 64, 128, 40
    shapes = {"wq": (H * hd, d), "wk": (Hkv * hd, d), "wv": (Hkv * hd, d), "wo": (d, H * hd), "w1": (dff, d), "wu": (dff, d), "w2": (d, dff)}
    raw = {name: o.synth_q1(rng, out_f, in_f // 128) for name, (out_f, in_f) in shapes.items()}
    w = {name: [q1_gpu.q1_register_weight(b, s.astype(np.int32))] for name, (b, s) in raw.items()}
    head_bits, head_scale = o.synth_q1(rng, vocab, d // 128)
    w["out_head"], w["out_head_vocab"] = q1_gpu.q1_register_weight(head_bits, head_scale.astype(np.int32)), vocab
    gains = {name: rng.integers(1 << 15, 1 << 17, size=n, dtype=np.int64) for name, n in (("n1g", d), ("n2g", d), ("qng", hd), ("kng", hd))}
    gh = {name: [q1_gpu.buf_upload_i64(g)] for name, g in gains.items()}
    cos, sin = o.build_rope_tables(T, hd, frac=16)
    gh["finalg"], gh["cos_h"], gh["sin_h"] = q1_gpu.buf_upload_i64(gains["n1g"]), q1_gpu.buf_upload_i64(cos), q1_gpu.buf_upload_i64(sin)
    x = rng.integers(-(1 << 14), 1 << 14, size=(T, d), dtype=np.int64)
    got = q1_gpu.prefill_forward_gpu(x, (T, d, 1, H, Hkv, hd, dff), w, gh, 16, 1, round((1 << 16) / 8), export_kv=True)
    assert got is not None
    want = onat.q1_linear(o.rmsnorm_fixed(x, 16, 1, gains["n1g"]), *raw["wv"], 16)
    assert np.array_equal(got[2][0, 0], want)
    q1_gpu.q1_free_weights()


def test_buffers_of_a_long_prompt_go_with_the_call():
    """600 rows with a feed-forward width of 65536 need 632 MB of activation rows, beyond what a call keeps; all of it is given back with
    the weights."""
    import torch

    from integer_inference_engine_b200 import q1_gpu
    rng = np.random.default_rng(1)
    d, H, Hkv, hd, dff, vocab, T = 128, 2, 1, 64, 65536, 40, 600
    shapes = {"wq": (H * hd, d), "wk": (Hkv * hd, d), "wv": (Hkv * hd, d), "wo": (d, H * hd), "w1": (dff, d), "wu": (dff, d), "w2": (d, dff)}
    x = rng.integers(-(1 << 14), 1 << 14, size=(T, d), dtype=np.int64)

    def prompt(rows):
        w = {}
        for name, (out_f, in_f) in shapes.items():
            bits, scale = o.synth_q1(np.random.default_rng(len(name)), out_f, in_f // 128)
            w[name] = [q1_gpu.q1_register_weight(bits, scale.astype(np.int32))]
        bits, scale = o.synth_q1(rng, vocab, 1)
        w["out_head"], w["out_head_vocab"] = q1_gpu.q1_register_weight(bits, scale.astype(np.int32)), vocab
        gh = {name: [q1_gpu.buf_upload_i64(np.full(n, 1 << 16, np.int64))] for name, n in (("n1g", d), ("n2g", d), ("qng", hd), ("kng", hd))}
        cos, sin = o.build_rope_tables(T, hd, frac=16)
        gh["finalg"], gh["cos_h"], gh["sin_h"] = q1_gpu.buf_upload_i64(np.full(d, 1 << 16, np.int64)), q1_gpu.buf_upload_i64(cos), q1_gpu.buf_upload_i64(sin)
        assert q1_gpu.prefill_forward_gpu(x[:rows], (rows, d, 1, H, Hkv, hd, dff), w, gh, 16, 1, 1 << 13) is not None

    q1_gpu.q1_free_weights()
    prompt(8)
    before = torch.cuda.mem_get_info()[0]
    prompt(T)
    kept = before - torch.cuda.mem_get_info()[0]
    assert kept < 450 << 20, kept                                       # the shared digit planes (315 MB) and attention scratch
    q1_gpu.q1_free_weights()
    assert before - torch.cuda.mem_get_info()[0] < 64 << 20


@pytest.mark.parametrize(("H", "Hkv", "positions"), [(8, 1, (0, 31, 32, 1000, 2300)), (4, 2, (127, 128, 129, 5)), (8, 1, (16384, 3, 700)), (32, 2, (70, 0, 40))])
def test_sequences_at_their_own_positions(H, Hkv, positions):
    """One decode step of sequences of very different lengths (in the one launch for all of them the shorter ones leave warps and CTAs of their
    clusters without keys), beyond the keys that launch takes, and with more query heads per KV head than it takes; against the checker."""
    from integer_inference_engine_b200 import q1_gpu
    from integer_inference_engine_b200.model import rope_tables
    from oracle import model_oracle
    rng = np.random.default_rng(sum(positions))
    d, hd, dff, vocab, B, cap = 256, 64, 128, 96, len(positions), max(positions) + 2
    qd, kd, inv_sqrt = H * hd, Hkv * hd, 1 << 13
    q1 = lambda out_f, in_f: o.synth_q1(rng, out_f, in_f // 128)
    raw = {"wqkv": q1(qd + 2 * kd, d), "wo": q1(d, qd), "w1u": q1(2 * dff, d), "w2": q1(d, dff)}
    top = {"embed": q1(vocab, d), "head": q1(vocab, d), "out_gain": rng.integers(1 << 15, 1 << 17, size=d, dtype=np.int64)}
    gains = {n: rng.integers(1 << 15, 1 << 17, size=s, dtype=np.int64) for n, s in (("n1", d), ("n2", d), ("qn", hd), ("kn", hd))}
    cos, sin = (np.ascontiguousarray(t, np.int64) for t in rope_tables(cap, hd, 1e6, 16))
    rows = {"wq": ("wqkv", 0, qd), "wk": ("wqkv", qd, qd + kd), "wv": ("wqkv", qd + kd, qd + 2 * kd), "wo": ("wo", 0, d), "w1": ("w1u", 0, dff),
            "wu": ("w1u", dff, 2 * dff), "w2": ("w2", 0, d)}
    w = {n: [q1_gpu.q1_register_weight(raw[m][0][a:b], raw[m][1][a:b].astype(np.int32))] for n, (m, a, b) in rows.items()}
    w["out_head"], w["out_head_vocab"] = q1_gpu.q1_register_weight(top["head"][0], top["head"][1].astype(np.int32)), vocab
    gh = {n: [q1_gpu.buf_upload_i64(gains[m])] for n, m in (("n1g", "n1"), ("n2g", "n2"), ("qng", "qn"), ("kng", "kn"))}
    gh["finalg"], gh["cos_h"], gh["sin_h"] = (q1_gpu.buf_upload_i64(a) for a in (top["out_gain"], cos, sin))
    ctx = q1_gpu.decode_ctx_create((B, 1, H, Hkv, hd, d, dff, vocab), w, gh, 16, 1, inv_sqrt, cap)
    assert ctx is not None
    caches = [[rng.integers(-(1 << 17), 1 << 17, size=(Hkv, cap, hd), dtype=np.int64) for _ in range(2)] for _ in range(B)]
    for b, pos in enumerate(positions):
        assert q1_gpu.decode_ctx_seed_seq(ctx, b, caches[b][0][None, :, :pos], caches[b][1][None, :, :pos])
    tokens = rng.integers(0, vocab, size=(2, B))
    cfg = dict(d=d, H=H, Hkv=Hkv, hd=hd, ffn=dff, frac=16)
    for step in range(2):
        x = np.concatenate([model_oracle.q1_rows(*top["embed"], int(t)) for t in tokens[step]])
        logits = q1_gpu.decode_step(ctx, x, [p + step for p in positions], vocab)
        assert logits is not None
        for b, pos in enumerate(positions):
            layer = dict(raw, **gains, k=caches[b][0], v=caches[b][1])
            _, _, want = model_oracle.q1_decode_token(int(tokens[step][b]), pos + step, [layer], top, cfg, cos, sin)
            assert np.array_equal(logits[b], want), (step, b)
    q1_gpu.decode_ctx_free(ctx)
    q1_gpu.q1_free_weights()
