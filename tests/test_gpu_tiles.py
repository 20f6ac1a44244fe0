"""Products of two rows and more on the tensor-core tiles against the CPU oracle, where the tiles can go wrong: row counts around
the tile widths, matrix rows around 128, one to many super-blocks (the sub-block sums are padded to four), three to eight
activation digits, both block formats, extreme scale patterns, uneven expert groups with experts that get no row."""
import numpy as np
import pytest

from oracle import native as onat
from oracle import qk_oracle as o

pytestmark = pytest.mark.gpu
FA, FW = 16, 24


@pytest.fixture(autouse=True)
def _from_two_rows():
    from integer_inference_engine_b200 import qk_cuda
    assert qk_cuda.available(), "CUDA library or GPU missing"
    qk_cuda.load_library().iie_set_tc_min_tokens(2)
    yield
    qk_cuda.free_all()


@pytest.mark.parametrize("qtype", [o.Q4_K, o.Q6_K])
@pytest.mark.parametrize("out_f,nb,T,xbits", [(8, 1, 2, 20), (128, 1, 16, 22), (129, 2, 17, 22), (120, 3, 32, 22), (200, 5, 33, 29), (264, 8, 31, 38),
                                              (130, 4, 65, 46), (72, 9, 5, 62), (2056, 1, 300, 22)])
def test_dense_tiles_match_the_oracle(qtype, out_f, nb, T, xbits):
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    rng = np.random.default_rng(out_f + nb * 5 + T)
    raw = np.frombuffer((o.synth_q4k if qtype == o.Q4_K else o.synth_q6k)(rng, out_f, nb), np.uint8).copy().reshape(out_f * nb, -1)
    fill = slice(4, 144) if qtype == o.Q4_K else slice(0, 208)                 # every scale, minimum and code at its largest in some blocks
    raw[::3, fill] = 0xFF
    if qtype == o.Q6_K:
        raw[1::3, 192:208] = 0x80                                             # scales of -128
    raw = raw.tobytes()
    x = rng.integers(-(1 << xbits), 1 << xbits, size=(T, nb * 256), dtype=np.int64)
    if xbits == 22:
        x[0], x[-1] = 8355711, -8421504                                        # the ends of three balanced digits
    device.read_flags()
    h = qk_cuda.register_weight(raw, out_f, nb, qtype)
    before = device.prefill_launch_counts()
    got = device.apply(h, torch.from_numpy(x).cuda(), out_f, FW).cpu().numpy()
    assert sum(device.prefill_launch_counts()) == sum(before) + 1, "the product did not run on the tiles"
    assert device.read_flags() == 0
    assert np.array_equal(got, onat.qk_linear(raw, x, out_f, nb, FW, qtype))


@pytest.mark.parametrize("qtype", [o.Q4_K, o.Q6_K])
@pytest.mark.parametrize("out_f,nb,T,xbits", [(128, 2, 2, 20), (1928, 8, 16, 22), (1900, 9, 5, 22), (264, 16, 64, 22), (264, 16, 64, 30), (520, 7, 100, 62), (9400, 3, 9, 22)])
def test_tiles_shared_by_clusters_match_the_oracle(qtype, out_f, nb, T, xbits):
    """Few tiles: two, four or eight CTAs share a tile's super-blocks (even and odd numbers of them), also where more digits than expected
    make the tiles narrower and a cluster walks several."""
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    rng = np.random.default_rng(out_f + nb * 7 + T)
    raw = np.frombuffer((o.synth_q4k if qtype == o.Q4_K else o.synth_q6k)(rng, out_f, nb), np.uint8).tobytes()
    x = rng.integers(-(1 << xbits), 1 << xbits, size=(T, nb * 256), dtype=np.int64)
    device.read_flags()
    h = qk_cuda.register_weight(raw, out_f, nb, qtype)
    got = device.apply(h, torch.from_numpy(x).cuda(), out_f, FW).cpu().numpy()
    assert device.read_flags() == 0
    assert np.array_equal(got, onat.qk_linear(raw, x, out_f, nb, FW, qtype))


@pytest.mark.parametrize("out_f,nb,T,xbits", [(4700, 3, 47, 30), (4700, 3, 47, 38), (6200, 3, 49, 30), (6200, 5, 49, 38), (2500, 8, 130, 30), (2500, 9, 130, 38)])
def test_narrow_and_wide_tiles_of_four_and_five_digits(out_f, nb, T, xbits):
    """Q6_K rows of four and five digits on either side of a wave of narrow tiles, over several super-blocks."""
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    rng = np.random.default_rng(out_f + nb + T)
    raw = o.synth_q6k(rng, out_f, nb)
    x = rng.integers(-(1 << xbits), 1 << xbits, size=(T, nb * 256), dtype=np.int64)
    device.read_flags()
    h = qk_cuda.register_weight(raw, out_f, nb, o.Q6_K)
    before = device.tile_form_counts()
    got = device.apply(h, torch.from_numpy(x).cuda(), out_f, FW).cpu().numpy()
    wide = (T + 15) // 16 * ((out_f + 127) // 128) > 148
    assert [b - a for a, b in zip(before, device.tile_form_counts())][1] == wide
    assert device.read_flags() == 0
    assert np.array_equal(got, onat.qk_linear(raw, x, out_f, nb, FW, o.Q6_K))


@pytest.mark.parametrize("qtype,out_f,nb,T,xbits,shared", [
    # the border in super-blocks saved, rows up to sixteen and above; the least and the most tiles that clusters share
    (o.Q4_K, 640, 2, 5, 22, 0), (o.Q4_K, 2048, 3, 5, 22, 0), (o.Q4_K, 1024, 4, 9, 22, 1), (o.Q4_K, 9472, 6, 16, 22, 1), (o.Q4_K, 9473, 6, 16, 22, 0), (o.Q4_K, 300, 3, 33, 22, 0),
    (o.Q6_K, 640, 2, 5, 22, 0), (o.Q6_K, 1024, 4, 9, 22, 0), (o.Q6_K, 200, 6, 2, 22, 1), (o.Q6_K, 9000, 8, 4, 22, 1), (o.Q6_K, 200, 8, 33, 22, 1), (o.Q6_K, 2048, 8, 100, 22, 0),
    # more digits than three: half of a cluster to a tile, or nobody shares; the wide Q6_K tiles of four digits, sixteen columns from five on
    (o.Q4_K, 1100, 8, 40, 30, 1), (o.Q4_K, 1100, 8, 40, 62, 1), (o.Q4_K, 4096, 8, 40, 30, 0), (o.Q6_K, 1100, 8, 40, 30, 1), (o.Q6_K, 1100, 8, 40, 38, 1), (o.Q6_K, 4090, 13, 40, 38, 0)])
def test_tiles_that_clusters_share(qtype, out_f, nb, T, xbits, shared):
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    rng = np.random.default_rng(out_f + nb * 3 + T)
    raw = np.frombuffer((o.synth_q4k if qtype == o.Q4_K else o.synth_q6k)(rng, out_f, nb), np.uint8).tobytes()
    x = rng.integers(-(1 << xbits), 1 << xbits, size=(T, nb * 256), dtype=np.int64)
    device.read_flags()
    h = qk_cuda.register_weight(raw, out_f, nb, qtype)
    before = device.tile_form_counts()
    got = device.apply(h, torch.from_numpy(x).cuda(), out_f, FW).cpu().numpy()
    assert device.tile_form_counts()[0] - before[0] == shared
    assert device.read_flags() == 0
    assert np.array_equal(got, onat.qk_linear(raw, x, out_f, nb, FW, qtype))


@pytest.mark.parametrize("down_q", [o.Q4_K, o.Q6_K])
@pytest.mark.parametrize("d,eff,E,k,T,mult", [(256, 256, 5, 2, 3, 1), (512, 256, 40, 1, 2, 1), (768, 512, 6, 3, 70, 1), (256, 768, 3, 3, 33, 200), (2304, 256, 24, 4, 48, 1),
                                                 (768, 512, 40, 2, 90, 200), (512, 256, 17, 2, 9, 20000)])
def test_expert_tiles_match_the_oracle(down_q, d, eff, E, k, T, mult):
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    rng = np.random.default_rng(d + eff + T)
    q4 = lambda r, c: o.synth_q4k(rng, r, c // 256)
    router, gate, up = q4(E, d), [q4(eff, d) for _ in range(E)], [q4(eff, d) for _ in range(E)]
    down = [(o.synth_q4k if down_q == o.Q4_K else o.synth_q6k)(rng, d, eff // 256) for _ in range(E)]
    h = o.to_fixed(rng.standard_normal((T, d)), FA) * mult
    reg = lambda w, r, c, q=o.Q4_K: qk_cuda.register_weight(w, r, c // 256, q)
    layer = device.MoELayer(reg(router, E, d), [reg(w, eff, d) for w in gate], [reg(w, eff, d) for w in up], [reg(w, d, eff, down_q) for w in down], k, d, eff)
    device.read_flags()
    out, ids, gates = layer.forward(torch.from_numpy(h).cuda(), FA, FW)
    torch.cuda.synchronize()
    assert device.read_flags() == 0
    ids_ref, gates_ref, out_ref = onat.moe_block(router, o.Q4_K, gate, up, down, o.Q4_K, down_q, k, h, d, eff, FA, FW)
    assert np.array_equal(ids.cpu().numpy(), ids_ref) and np.array_equal(gates.cpu().numpy(), gates_ref)
    assert np.array_equal(out.cpu().numpy(), out_ref)
    layer.close()


@pytest.mark.parametrize("T,distinct,eight", [(128, 1, 0), (128, 0, 1), (71, 1, 1), (73, 1, 0), (96, 2, 0), (40, 1, 1), (33, 0, 1)])
def test_gate_up_tiles_follow_the_routing(T, distinct, eight):
    """Tokens that all choose the same few experts (`distinct` different rows among them, 0: all) give those many rows each: tiles of sixteen rows.  Spread
    over the experts, or too few to fill the device, they have tiles of eight."""
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    rng = np.random.default_rng(T + distinct)
    d, eff, E, k = 256, 768, 128, 8
    q4 = lambda r, c: o.synth_q4k(rng, r, c // 256)
    router, gate, up, down = q4(E, d), [q4(eff, d) for _ in range(E)], [q4(eff, d) for _ in range(E)], [q4(d, eff) for _ in range(E)]
    h = o.to_fixed(rng.standard_normal((T, d)), FA)
    if distinct:
        h = h[np.arange(T) % distinct] + rng.integers(-3, 4, size=(T, d))      # the same experts, other values
    reg = lambda w, r, c: qk_cuda.register_weight(w, r, c // 256, o.Q4_K)
    layer = device.MoELayer(reg(router, E, d), [reg(w, eff, d) for w in gate], [reg(w, eff, d) for w in up], [reg(w, d, eff) for w in down], k, d, eff)
    device.read_flags()
    before, shapes = device.tile_form_counts()[2], sum(device.prefill_launch_counts())
    out, ids, gates = layer.forward(torch.from_numpy(h).cuda(), FA, FW)
    assert device.tile_form_counts()[2] - before == eight and sum(device.prefill_launch_counts()) - shapes == 3
    assert device.read_flags() == 0
    ids_ref, gates_ref, out_ref = onat.moe_block(router, o.Q4_K, gate, up, down, o.Q4_K, o.Q4_K, k, h, d, eff, FA, FW)
    assert np.array_equal(ids.cpu().numpy(), ids_ref) and np.array_equal(gates.cpu().numpy(), gates_ref)
    assert np.array_equal(out.cpu().numpy(), out_ref)
    layer.close()


def test_replays_of_a_short_graph_find_their_digit_count_cleared():
    """One product captured on its own: a replay over wide rows leaves the replays after it the digit planes that their rows need."""
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    rng = np.random.default_rng(8)
    raw = o.synth_q4k(rng, 256, 1)
    h = qk_cuda.register_weight(raw, 256, 1, o.Q4_K)
    x, out = torch.zeros((4, 256), dtype=torch.int64, device="cuda"), torch.empty((4, 256), dtype=torch.int64, device="cuda")
    device.read_flags()
    for _ in range(9):                                                  # eager calls between: every cell has been used
        device.apply(h, x, 256, 24, out=out)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        device.apply(h, x, 256, 24, out=out)
    for bits in (16, 50, 16, 16, 50, 50, 16):
        rows = rng.integers(-(1 << bits), 1 << bits, size=(4, 256), dtype=np.int64)
        x.copy_(torch.from_numpy(rows))
        before = device.prefill_launch_counts()
        graph.replay()
        torch.cuda.synchronize()
        ran = [b - a for a, b in zip(before, device.prefill_launch_counts())]
        assert ran[5 if bits == 16 else 7] == 1 and sum(ran) == 1, (bits, ran)
        assert np.array_equal(out.cpu().numpy(), onat.qk_linear(raw, rows, 256, 1, 24, o.Q4_K))
    assert device.read_flags() == 0
    del graph
    qk_cuda.free_all()


def test_launch_counts_fit_the_room_of_earlier_callers():
    import ctypes

    from integer_inference_engine_b200 import qk_cuda
    lib = qk_cuda.load_library()
    buf = (ctypes.c_uint64 * 8)(*[77] * 8)
    assert lib.iie_prefill_launch_counts(buf, 6) == -1
    assert lib.iie_prefill_launch_counts(buf, 7) == 7 and buf[7] == 77
    assert lib.iie_prefill_launch_counts(buf, 8) == 8 and buf[7] != 77


@pytest.mark.parametrize("qtype", [o.Q4_K, o.Q6_K])
@pytest.mark.parametrize("T", [2, 33])
def test_largest_sums_of_a_row(qtype, T):
    """64 super-blocks of the largest scales, minima and codes at the largest block scales the tiles take, every value at one end of its digits."""
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    out_f, nb = 16, 64
    raw = np.zeros((out_f, nb, 144 if qtype == o.Q4_K else 210), np.uint8)
    raw[:, :, slice(4, 144) if qtype == o.Q4_K else slice(0, 208)] = 0xFF
    raw[1::4, :, 16 if qtype == o.Q4_K else 0:144 if qtype == o.Q4_K else 192] = 0            # the smallest codes
    if qtype == o.Q6_K:
        raw[::2, :, 192:208] = 0x80                                            # scales of -128
    half = lambda v: np.frombuffer(np.float16(v).tobytes(), np.uint8)
    if qtype == o.Q4_K:
        raw[:, :, 0:2], raw[:, :, 2:4] = half(0.49975586), half(3.9980469)     # d below 2^23, dmin below 2^26 at 2^24
    else:
        raw[:, :, 208:210] = half(0.49975586)
    buf = raw.tobytes()
    h = qk_cuda.register_weight(buf, out_f, nb, qtype)
    device.read_flags()
    for top, bottom in ((8355711, -8421504), (0x7F7F7F7F, -0x80808080), (0x7F7F7F7F7F7F, -0x808080808080), (0x7F7F7F7F7F7F7F7F, -0x7F7F7F7F7F7F7F7F)):
        x = np.full((T, nb * 256), bottom, np.int64)
        x[1::2] = top
        before = device.prefill_launch_counts()
        got = device.apply(h, torch.from_numpy(x).cuda(), out_f, FW).cpu().numpy()
        assert sum(device.prefill_launch_counts()) == sum(before) + 1, "the product did not run on the tiles"
        assert np.array_equal(got, onat.qk_linear(buf, x, out_f, nb, FW, qtype))
    assert device.read_flags() == 0


@pytest.mark.parametrize("fa", [1, 5, 12, 20, 24, 25])
def test_expert_tiles_at_other_activation_scales(fa):
    """The epilogue's 32-bit SiLU up to a scale of 2^24, the general one beyond; gates of all magnitudes around the sigmoid's clip."""
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    rng = np.random.default_rng(fa)
    d, eff, E, k, T = 256, 256, 2, 2, 40
    q4 = lambda r, c: o.synth_q4k(rng, r, c // 256)
    router, gate, up, down = q4(E, d), [q4(eff, d) for _ in range(E)], [q4(eff, d) for _ in range(E)], [q4(d, eff) for _ in range(E)]
    h = np.rint(rng.standard_normal((T, d)) * np.exp2(rng.uniform(-3, 9, size=(T, 1))) * (1 << fa)).astype(np.int64)
    reg = lambda w, r, c: qk_cuda.register_weight(w, r, c // 256, o.Q4_K)
    layer = device.MoELayer(reg(router, E, d), [reg(w, eff, d) for w in gate], [reg(w, eff, d) for w in up], [reg(w, d, eff) for w in down], k, d, eff)
    device.read_flags()
    before = device.prefill_launch_counts()
    out, ids, gates = layer.forward(torch.from_numpy(h).cuda(), fa, FW)
    torch.cuda.synchronize()
    assert sum(device.prefill_launch_counts()) - sum(before) == 3
    ids_ref, gates_ref, out_ref = onat.moe_block(router, o.Q4_K, gate, up, down, o.Q4_K, o.Q4_K, k, h, d, eff, fa, FW)
    assert device.read_flags() == 0
    assert np.array_equal(ids.cpu().numpy(), ids_ref) and np.array_equal(gates.cpu().numpy(), gates_ref)
    assert np.array_equal(out.cpu().numpy(), out_ref)
    layer.close()


@pytest.mark.parametrize("T", [3, 40])
def test_gate_values_of_the_least_int64(T):
    """A gate product of exactly -2^63, whose sigmoid is one half because its distance from zero wraps: both kinds of gate / up tiles."""
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    d, eff, E, k = 256, 256, 2, 2
    def one_weight(d_half, col, code):                                         # rows of one block: scale 1, `code` at one of the first 32 columns
        raw = np.zeros((eff, 144), np.uint8)
        raw[:, 0:2] = np.frombuffer(np.float16(d_half).tobytes(), np.uint8)
        raw[:, 4], raw[:, 16 + col] = 1, code
        return raw.tobytes()
    rng = np.random.default_rng(T)
    gate, up = [one_weight(0.25, 0, 8)] * E, [one_weight(0.125, 1, 1)] * E
    router, down = np.zeros((E, 144), np.uint8).tobytes(), [o.synth_q4k(rng, d, eff // 256) for _ in range(E)]
    h = o.to_fixed(rng.standard_normal((T, d)), FA)
    h[1, :2] = -(1 << 62), 1000                                                # gate -2^62 * 8 / 4, up 125
    reg = lambda w, r, c: qk_cuda.register_weight(w, r, c // 256, o.Q4_K)
    layer = device.MoELayer(reg(router, E, d), [reg(w, eff, d) for w in gate], [reg(w, eff, d) for w in up], [reg(w, d, eff) for w in down], k, d, eff)
    device.read_flags()
    before = device.tile_form_counts()[2]
    out, ids, gates = layer.forward(torch.from_numpy(h).cuda(), FA, FW)
    assert device.tile_form_counts()[2] - before == (T == 3)
    assert device.read_flags() == 0
    ids_ref, gates_ref, out_ref = onat.moe_block(router, o.Q4_K, gate, up, down, o.Q4_K, o.Q4_K, k, h, d, eff, FA, FW)
    assert np.any(out_ref[1] != 0)
    assert np.array_equal(ids.cpu().numpy(), ids_ref) and np.array_equal(gates.cpu().numpy(), gates_ref)
    assert np.array_equal(out.cpu().numpy(), out_ref)
    layer.close()


@pytest.mark.parametrize(("qtype", "out_f", "nb", "T", "tiles"), [(o.Q4_K, 40960, 1, 3, 0), (o.Q4_K, 40961, 1, 3, 1), (o.Q4_K, 300, 9, 2, 0), (o.Q4_K, 300, 9, 4, 1),
                                                                  (o.Q6_K, 5120, 8, 3, 0), (o.Q6_K, 5121, 8, 2, 1), (o.Q6_K, 64, 3, 4, 1), (o.Q4_K, 24, 48, 3, 1)])
def test_dense_products_by_size(qtype, out_f, nb, T, tiles):
    """Both sides of the border between the streaming kernel and the tiles, and a row length that only the tiles take."""
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    qk_cuda.load_library().iie_set_tc_min_tokens(0)
    rng = np.random.default_rng(out_f + T)
    raw = (o.synth_q4k if qtype == o.Q4_K else o.synth_q6k)(rng, out_f, nb)
    h = qk_cuda.register_weight(raw, out_f, nb, qtype)
    x = rng.integers(-(1 << 22), 1 << 22, size=(T, nb * 256), dtype=np.int64)
    device.read_flags()
    before = device.prefill_launch_counts()
    got = device.apply(h, torch.from_numpy(x).cuda(), out_f, FW).cpu().numpy()
    assert sum(device.prefill_launch_counts()) - sum(before) == tiles
    assert device.read_flags() == 0
    assert np.array_equal(got, onat.qk_linear(raw, x, out_f, nb, FW, qtype))


@pytest.mark.parametrize(("d", "eff", "E", "k", "T", "tiles"), [(256, 256, 4, 2, 3, 0), (256, 256, 4, 2, 4, 2), (256, 256, 4, 2, 191, 2), (256, 256, 4, 2, 192, 3),
                                                                (1024, 512, 2, 2, 127, 2), (1024, 512, 2, 2, 128, 3), (512, 256, 200, 1, 40, 2)])
def test_expert_blocks_by_size(d, eff, E, k, T, tiles):
    """The kernels of router, gate / up and down change one by one with the rows; the block's bytes do not."""
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    qk_cuda.load_library().iie_set_tc_min_tokens(0)
    rng = np.random.default_rng(d + E + T)
    q4 = lambda r, c: o.synth_q4k(rng, r, c // 256)
    router, gate, up = q4(E, d), [q4(eff, d) for _ in range(E)], [q4(eff, d) for _ in range(E)]
    down = [o.synth_q6k(rng, d, eff // 256) for _ in range(E)]
    h = o.to_fixed(rng.standard_normal((T, d)), FA)
    reg = lambda w, r, c, q=o.Q4_K: qk_cuda.register_weight(w, r, c // 256, q)
    layer = device.MoELayer(reg(router, E, d), [reg(w, eff, d) for w in gate], [reg(w, eff, d) for w in up], [reg(w, d, eff, o.Q6_K) for w in down], k, d, eff)
    device.read_flags()
    before = device.prefill_launch_counts()
    out, ids, gates = layer.forward(torch.from_numpy(h).cuda(), FA, FW)
    torch.cuda.synchronize()
    assert sum(device.prefill_launch_counts()) - sum(before) == tiles
    assert device.read_flags() == 0
    ids_ref, gates_ref, out_ref = onat.moe_block(router, o.Q4_K, gate, up, down, o.Q4_K, o.Q6_K, k, h, d, eff, FA, FW)
    assert np.array_equal(ids.cpu().numpy(), ids_ref) and np.array_equal(gates.cpu().numpy(), gates_ref)
    assert np.array_equal(out.cpu().numpy(), out_ref)
    layer.close()


@pytest.mark.parametrize("qtype", [o.Q4_K, o.Q6_K])
@pytest.mark.parametrize("T,xbits", [(9, 22), (9, 30), (16, 38), (9, 46), (9, 62), (130, 22), (130, 30), (130, 38)])
def test_dense_tiles_beyond_those_that_clusters_share(qtype, T, xbits):
    """The usual form over several super-blocks (their rings wrap; the minima of four share a row of sums), three to eight digits, narrow and wide
    tiles, extreme blocks among the others."""
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    out_f, nb = (9500, 6) if T <= 16 else (2500, 9)
    rng = np.random.default_rng(T + xbits)
    raw = np.frombuffer((o.synth_q4k if qtype == o.Q4_K else o.synth_q6k)(rng, out_f, nb), np.uint8).copy().reshape(out_f * nb, -1)
    raw[::5, slice(4, 144) if qtype == o.Q4_K else slice(0, 208)] = 0xFF
    if qtype == o.Q6_K:
        raw[1::5, 192:208] = 0x80
    raw = raw.tobytes()
    x = rng.integers(-(1 << xbits), 1 << xbits, size=(T, nb * 256), dtype=np.int64)
    device.read_flags()
    h = qk_cuda.register_weight(raw, out_f, nb, qtype)
    before, shared = device.prefill_launch_counts(), device.tile_form_counts()[0]
    got = device.apply(h, torch.from_numpy(x).cuda(), out_f, FW).cpu().numpy()
    assert sum(device.prefill_launch_counts()) == sum(before) + 1 and device.tile_form_counts()[0] == shared
    assert device.read_flags() == 0
    assert np.array_equal(got, onat.qk_linear(raw, x, out_f, nb, FW, qtype))


def _largest_blocks(qtype, rows, nb):
    """The largest scales, minima and codes at the largest block scales the tiles take, with the smallest codes in every fourth row."""
    raw = np.zeros((rows, nb, 144 if qtype == o.Q4_K else 210), np.uint8)
    raw[:, :, slice(4, 144) if qtype == o.Q4_K else slice(0, 208)] = 0xFF
    raw[1::4, :, 16 if qtype == o.Q4_K else 0:144 if qtype == o.Q4_K else 192] = 0
    half = lambda v: np.frombuffer(np.float16(v).tobytes(), np.uint8)
    if qtype == o.Q4_K:
        raw[:, :, 0:2], raw[:, :, 2:4] = half(0.49975586), half(3.9980469)     # d below 2^23, dmin below 2^26 at 2^24
    else:
        raw[::2, :, 192:208] = 0x80                                            # scales of -128
        raw[:, :, 208:210] = half(0.49975586)
    return raw


@pytest.mark.parametrize("qtype", [o.Q4_K, o.Q6_K])
@pytest.mark.parametrize("T", [2, 33])
def test_largest_sums_of_a_row_beyond_those_that_clusters_share(qtype, T):
    """64 super-blocks of the largest blocks in the usual form: sixteen rows of them, repeated over more tiles than clusters take."""
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    nb, repeat = 64, 600
    buf = _largest_blocks(qtype, 16, nb).tobytes()
    h = qk_cuda.register_weight(buf * repeat, 16 * repeat, nb, qtype)
    device.read_flags()
    for digits in (3, 4, 5, 6, 8):
        top = int.from_bytes(b"\x7f" * digits, "little")
        x = np.full((T, nb * 256), -top, np.int64)
        x[1::2] = top
        before, shared = device.prefill_launch_counts(), device.tile_form_counts()[0]
        got = device.apply(h, torch.from_numpy(x).cuda(), 16 * repeat, FW).cpu().numpy()
        assert sum(device.prefill_launch_counts()) == sum(before) + 1 and device.tile_form_counts()[0] == shared
        want = onat.qk_linear(buf, x[:2], 16, nb, FW, qtype)
        assert np.array_equal(got.reshape(T, repeat, 16), np.broadcast_to(want[np.arange(T) % 2][:, None], (T, repeat, 16)))
    assert device.read_flags() == 0
    qk_cuda.free_all()


@pytest.mark.parametrize("digits", [3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("T", [3, 8])
def test_largest_sums_of_the_eight_row_tiles(digits, T):
    """Gate / up over 64 super-blocks of the largest blocks, every value at one end of its digits: the 32-bit sums of a super-block and both walks at
    their limits.  Successive super-blocks have opposite signs and the last two ordinary values, so that the products stay in range."""
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    d, eff, E, k, nb = 64 * 256, 256, 2, 2, 64
    rng = np.random.default_rng(digits)
    weights = []
    for _ in range(2 * E):
        raw = _largest_blocks(o.Q4_K, eff, nb)
        raw[:, 62:] = np.frombuffer(o.synth_q4k(rng, eff, 2), np.uint8).reshape(eff, 2, 144)
        raw[:, 2] = np.frombuffer(o.synth_q4k(rng, eff, 1), np.uint8).reshape(eff, 144)      # and a pair of another scale
        raw[:, 3] = raw[:, 2]
        weights.append(raw.tobytes())
    gate, up, router = weights[:E], weights[E:], np.zeros((E * nb, 144), np.uint8).tobytes()
    down = [o.synth_q4k(rng, d, eff // 256) for _ in range(E)]
    top = int.from_bytes(b"\x7f" * digits, "little")
    h = np.full((T, nb, 256), top, np.int64)
    h[:, 1::2] = -top
    h[1::3] = -h[1::3]
    h[2::3, :, ::2] = 0
    h[:, 62:] = rng.integers(-(1 << 17), 1 << 17, size=(T, 2, 256))
    h = h.reshape(T, d)
    reg = lambda w, r, c: qk_cuda.register_weight(w, r, c // 256, o.Q4_K)
    layer = device.MoELayer(reg(router, E, d), [reg(w, eff, d) for w in gate], [reg(w, eff, d) for w in up], [reg(w, d, eff) for w in down], k, d, eff)
    device.read_flags()
    before = device.tile_form_counts()[2]
    out, ids, gates = layer.forward(torch.from_numpy(h).cuda(), FA, FW)
    assert device.tile_form_counts()[2] - before == 1
    assert device.read_flags() == 0
    ids_ref, gates_ref, out_ref = onat.moe_block(router, o.Q4_K, gate, up, down, o.Q4_K, o.Q4_K, k, h, d, eff, FA, FW)
    assert np.array_equal(ids.cpu().numpy(), ids_ref) and np.array_equal(gates.cpu().numpy(), gates_ref)
    assert np.array_equal(out.cpu().numpy(), out_ref)
    layer.close()


@pytest.mark.parametrize("fa", [1, 5, 12, 20, 24, 25])
def test_eight_row_tiles_at_other_activation_scales(fa):
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    rng = np.random.default_rng(fa)
    d, eff, E, k, T = 256, 256, 5, 2, 17
    q4 = lambda r, c: o.synth_q4k(rng, r, c // 256)
    router, gate, up, down = q4(E, d), [q4(eff, d) for _ in range(E)], [q4(eff, d) for _ in range(E)], [q4(d, eff) for _ in range(E)]
    h = np.rint(rng.standard_normal((T, d)) * np.exp2(rng.uniform(-3, 9, size=(T, 1))) * (1 << fa)).astype(np.int64)
    reg = lambda w, r, c: qk_cuda.register_weight(w, r, c // 256, o.Q4_K)
    layer = device.MoELayer(reg(router, E, d), [reg(w, eff, d) for w in gate], [reg(w, eff, d) for w in up], [reg(w, d, eff) for w in down], k, d, eff)
    device.read_flags()
    before = device.tile_form_counts()[2]
    out, ids, gates = layer.forward(torch.from_numpy(h).cuda(), fa, FW)
    assert device.tile_form_counts()[2] - before == 1
    ids_ref, gates_ref, out_ref = onat.moe_block(router, o.Q4_K, gate, up, down, o.Q4_K, o.Q4_K, k, h, d, eff, fa, FW)
    assert device.read_flags() == 0
    assert np.array_equal(ids.cpu().numpy(), ids_ref) and np.array_equal(gates.cpu().numpy(), gates_ref)
    assert np.array_equal(out.cpu().numpy(), out_ref)
    layer.close()


@pytest.mark.parametrize("T,eight", [(5, 0), (6, 1), (64, 1), (65, 0)])      # 591 and 658 of 650
def test_eight_row_tiles_by_size(T, eight):
    """Both borders of the eight-row tiles: the experts that are met have tiles for the device, eight rows per expert."""
    import torch

    from integer_inference_engine_b200 import device, qk_cuda
    qk_cuda.load_library().iie_set_tc_min_tokens(0)
    rng = np.random.default_rng(T)
    d, eff, E, k = 1024, 768, 32, 4
    q4 = lambda r, c: o.synth_q4k(rng, r, c // 256)
    router, gate, up = q4(E, d), [q4(eff, d) for _ in range(E)], [q4(eff, d) for _ in range(E)]
    down = [o.synth_q6k(rng, d, eff // 256) for _ in range(E)]
    h = o.to_fixed(rng.standard_normal((T, d)), FA)
    reg = lambda w, r, c, q=o.Q4_K: qk_cuda.register_weight(w, r, c // 256, q)
    layer = device.MoELayer(reg(router, E, d), [reg(w, eff, d) for w in gate], [reg(w, eff, d) for w in up], [reg(w, d, eff, o.Q6_K) for w in down], k, d, eff)
    device.read_flags()
    before = device.tile_form_counts()[2]
    out, ids, gates = layer.forward(torch.from_numpy(h).cuda(), FA, FW)
    assert device.tile_form_counts()[2] - before == eight
    assert device.read_flags() == 0
    ids_ref, gates_ref, out_ref = onat.moe_block(router, o.Q4_K, gate, up, down, o.Q4_K, o.Q6_K, k, h, d, eff, FA, FW)
    assert np.array_equal(ids.cpu().numpy(), ids_ref) and np.array_equal(gates.cpu().numpy(), gates_ref)
    assert np.array_equal(out.cpu().numpy(), out_ref)
    layer.close()
