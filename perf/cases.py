"""What this framework is measured on: the calls its users make, at the shapes of its own configurations.

Two models stand behind the cases, both with seeded synthetic weights of the distributions in
``integer_inference_engine_b200/synth.py`` and ``q1_model.py``:

* the 30B-A3B mixture-of-experts decoder (48 blocks, width 2048, 32 query and 4 KV heads of 128, 128 experts of 768, eight
  per token, Q4_K matrices, Q6_K down projections and tied head, vocabulary 151936);
* the 8B 1-bit decoder (Q1_0, width 4096, 32 query and 8 KV heads of 128, feed-forward width 12288).

Weights are registered once per process, as a serving program does, and shared by the states; a state has its own inputs.
All results are integers defined bit for bit, so every case is compared exactly.
"""
from __future__ import annotations

import functools
import math
import weakref

import numpy as np
import torch

from integer_inference_engine_b200 import device, ep_model, model, q1_gpu, q1_model, qk_cuda, synth
from integer_inference_engine_b200.qk_cuda import Q4_K

FA, FW, FRAC = 16, 24, 16
D, H, HKV, HD, EFF, EXPERTS, TOP_K, VOCAB, BLOCKS, WINDOW = 2048, 32, 4, 128, 768, 128, 8, 151936, 48, 4096
QD, KD, NB = H * HD, HKV * HD, D // 256
STEP_BLOCKS = 4                                    # blocks of the batched step: 1.6 GB of expert weights, far beyond L2
Q_D, Q_H, Q_HKV, Q_HD, Q_FFN, Q_BLOCKS = 4096, 32, 8, 128, 12288, 36
Q_HOST_BLOCKS = 12                                 # blocks of the 1-bit model driven through host arrays: 0.4 GB
Q_ROWS = 640                                       # cache rows and rotation table of the 1-bit model
ATTN_SETS = 8                                      # attention matrices of a prefill: drawn so that q, k, v are of order one


def listed():
    return [
        # interactive generation, one token per call: a long conversation and a young one
        {"name": "decode_4096", "kind": "decode", "context": 4096},
        {"name": "decode_300", "kind": "decode", "context": 300},
        # serving: one token for every running sequence, a full batch and a nearly idle server
        {"name": "step_64x4096", "kind": "step", "sequences": 64, "context": 4096},
        {"name": "step_7x1500", "kind": "step", "sequences": 7, "context": 1500},
        # prompt processing of one block: a long prompt, a ragged later chunk of one (no rotation, as every fourth block),
        # and a short question
        {"name": "prefill_2048", "kind": "prefill", "tokens": 2048, "start": 0, "rope": True},
        {"name": "prefill_333_at_2900", "kind": "prefill", "tokens": 333, "start": 2900, "rope": False},
        {"name": "prefill_45", "kind": "prefill", "tokens": 45, "start": 0, "rope": True},
        # the drop-in host-array calls of an engine that keeps its activations in NumPy: a MoE block of 16 rows, and the
        # smallest call there is, the Q, K and V products of one row
        {"name": "moe_host_16", "kind": "moe_host", "tokens": 16},
        {"name": "qkv_host_1", "kind": "qkv_host", "tokens": 1},
        # the 1-bit model: a token of interactive generation, a prompt, and one token for six sequences at their own positions
        {"name": "q1_decode_512", "kind": "q1_decode", "context": 512},
        {"name": "q1_prefill_512", "kind": "q1_prefill", "tokens": 512, "export": False},
        {"name": "q1_step_6", "kind": "q1_step", "sequences": 6, "context": 200},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "step", "prefill", "prefill", "moe_host", "qkv_host", "q1_decode", "q1_prefill", "q1_step"])
    if kind == "decode":
        return {"kind": kind, "context": _log(rng, 64, 4096)}
    if kind == "step":
        return {"kind": kind, "sequences": _log(rng, 2, 64), "context": _log(rng, 256, 4096)}
    if kind == "prefill":
        tokens = _log(rng, 16, 2048)
        start = rng.choice([0, rng.randrange(1, 4096 - tokens)])
        # a later chunk of the longest prompts would cost more than the longest listed prompt
        return {"kind": kind, "tokens": tokens, "start": start if tokens <= 1024 else 0, "rope": rng.random() < 0.75}
    if kind == "moe_host":
        return {"kind": kind, "tokens": _log(rng, 1, 64)}
    if kind == "qkv_host":
        return {"kind": kind, "tokens": _log(rng, 1, 32)}
    if kind == "q1_decode":
        return {"kind": kind, "context": _log(rng, 32, 600)}
    if kind == "q1_prefill":
        return {"kind": kind, "tokens": _log(rng, 12, 512), "export": rng.random() < 0.5}
    return {"kind": kind, "sequences": _log(rng, 1, 12), "context": _log(rng, 32, 256)}


# ------------------------------------------------------------------------------------------- models, once per process ---
@functools.lru_cache(maxsize=1)
def moe_model():
    return model.SyntheticDecoder(n_layers=BLOCKS, d_model=D, n_heads=H, n_kv=HKV, head_dim=HD, e_ffn=EFF, n_experts=EXPERTS,
                                  top_k=TOP_K, vocab=VOCAB, context=8, max_new=WINDOW + 8, window=WINDOW, fa=FA, fw=FW)


@functools.lru_cache(maxsize=1)
def attention_weights():
    """Attention matrices for the block-wise calls: the fused Q/K/V matrix, its three parts on their own, and O."""
    out = []
    for i in range(ATTN_SETS):
        gen = torch.Generator(device="cuda").manual_seed(4001 + i)
        raw = synth.synth_q4k((QD + 2 * KD) * NB, gen, 2e-4).view(QD + 2 * KD, NB * 144)
        part = lambda a, b: device.register_weight(raw[a:b].contiguous().view(-1), b - a, NB, Q4_K)
        wo = device.register_weight(synth.synth_q4k(D * (QD // 256), gen, 2e-4).view(-1), D, QD // 256, Q4_K)
        out.append({"wqkv": part(0, QD + 2 * KD), "wq": part(0, QD), "wk": part(QD, QD + KD), "wv": part(QD + KD, QD + 2 * KD),
                    "wo": wo})
    return out


@functools.lru_cache(maxsize=1)
def step_model(sequences, context):
    return ep_model.ExpertParallelDecoder(sequences, n_layers=STEP_BLOCKS, d_model=D, n_heads=H, n_kv=HKV, head_dim=HD, e_ffn=EFF,
                                          n_experts=EXPERTS, top_k=TOP_K, vocab=VOCAB, context=context, max_new=4, window=WINDOW,
                                          fa=FA, fw=FW)


def _q1_weight(out_f, in_f, gen):
    bits = torch.randint(0, 256, (out_f, in_f // 128, 16), generator=gen, device="cuda", dtype=torch.uint8)
    scale = (torch.randn((out_f, in_f // 128), generator=gen, device="cuda").abs() * 0.02).to(torch.float16)
    return bits.cpu().numpy(), torch.round(scale.double() * (1 << FRAC)).to(torch.int32).cpu().numpy()


def _q1_gain(n, gen):
    return torch.round((torch.randn(n, generator=gen, device="cuda", dtype=torch.float64).abs() + 0.5) * (1 << FRAC)).to(torch.int64).cpu().numpy()


@functools.lru_cache(maxsize=1)
def q1_decoder():
    gen = torch.Generator(device="cuda").manual_seed(5001)
    qd, kd = Q_H * Q_HD, Q_HKV * Q_HD
    cache = lambda: torch.randint(-(1 << 17), 1 << 17, (Q_HKV, Q_ROWS, Q_HD), generator=gen, device="cuda", dtype=torch.int32)
    layers = ({"n1": _q1_gain(Q_D, gen), "n2": _q1_gain(Q_D, gen), "qn": _q1_gain(Q_HD, gen), "kn": _q1_gain(Q_HD, gen),
               "wqkv": _q1_weight(qd + 2 * kd, Q_D, gen), "wo": _q1_weight(Q_D, qd, gen), "w1u": _q1_weight(2 * Q_FFN, Q_D, gen),
               "w2": _q1_weight(Q_D, Q_FFN, gen), "k": cache(), "v": cache()} for _ in range(Q_BLOCKS))
    top = {"embed": _q1_weight(VOCAB, Q_D, gen), "head": _q1_weight(VOCAB, Q_D, gen), "out_gain": _q1_gain(Q_D, gen)}
    cos, sin = model.rope_tables(Q_ROWS, Q_HD, 1e6, FRAC)
    return q1_model.Q1Decoder(Q_D, Q_H, Q_HKV, Q_HD, Q_FFN, VOCAB, layers, top, cos, sin, 0, FRAC)


@functools.lru_cache(maxsize=1)
def q1_host_model():
    """Weight and gain handles as the 1-bit engine hands them to the whole-model calls."""
    gen = torch.Generator(device="cuda").manual_seed(6001)
    qd, kd = Q_H * Q_HD, Q_HKV * Q_HD
    shapes = {"wq": (qd, Q_D), "wk": (kd, Q_D), "wv": (kd, Q_D), "wo": (Q_D, qd), "w1": (Q_FFN, Q_D), "wu": (Q_FFN, Q_D), "w2": (Q_D, Q_FFN)}
    gains = {"n1g": Q_D, "n2g": Q_D, "qng": Q_HD, "kng": Q_HD}
    w = {name: [q1_gpu.q1_register_weight(*_q1_weight(*shape, gen)) for _ in range(Q_HOST_BLOCKS)] for name, shape in shapes.items()}
    g = {name: [q1_gpu.buf_upload_i64(_q1_gain(n, gen)) for _ in range(Q_HOST_BLOCKS)] for name, n in gains.items()}
    w["out_head"], w["out_head_vocab"] = q1_gpu.q1_register_weight(*_q1_weight(VOCAB, Q_D, gen)), VOCAB
    cos, sin = model.rope_tables(Q_ROWS, Q_HD, 1e6, FRAC)
    g["finalg"], g["cos_h"], g["sin_h"] = q1_gpu.buf_upload_i64(_q1_gain(Q_D, gen)), q1_gpu.buf_upload_i64(cos), q1_gpu.buf_upload_i64(sin)
    return w, g


# ------------------------------------------------------------------------------------------------------------- states ---
class State(dict):
    """Inputs of one case; a dict that can carry a finaliser."""
    __hash__ = object.__hash__


def _pinned_token(token):
    return torch.tensor([token], dtype=torch.int32).pin_memory()


def _rows(tokens, width, gen):
    return torch.round(torch.randn((tokens, width), generator=gen, device="cuda", dtype=torch.float64) * (1 << FA)).to(torch.int64)


def prepare(case, seed):
    kind = case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    cache = lambda *shape: torch.randint(-(1 << 18), 1 << 18, shape, generator=gen, device="cuda", dtype=torch.int32)
    s = State(kind=kind)
    if kind == "decode":
        # a conversation of its own on the shared weights: its caches, its captured step
        m, context = moe_model(), case["context"]
        rows = context + 8
        attn = [{"wqkv": a["wqkv"], "wo": a["wo"], "k": cache(HKV, rows, HD), "v": cache(HKV, rows, HD)} for a in m.attn]
        s["decoder"] = model.Decoder(d_model=D, n_heads=H, n_kv=HKV, head_dim=HD, top_k=TOP_K, vocab=VOCAB, window=WINDOW, fa=FA, fw=FW,
                                     attn=attn, moe_layers=m.moe_layers, gain_handles=m.gain_handles, embd=m.embd,
                                     out_gain_h=m.out_gain_h, cos=m.cos[:rows], sin=m.sin[:rows], position=context)
        s["decoder"].capture(context)
        s["context"], s["token"], s["next"] = context, _pinned_token(int(rng.integers(VOCAB))), _pinned_token(0)
    elif kind == "step":
        s["decoder"] = step_model(case["sequences"], case["context"])
        s["tokens"] = torch.randint(0, VOCAB, (case["sequences"],), generator=gen, device="cuda", dtype=torch.int32)
    elif kind == "prefill":
        tokens, start, m = case["tokens"], case["start"], moe_model()
        at = int(rng.integers(BLOCKS))
        s.update(tokens=tokens, start=start, rope=1 if case["rope"] else 0, layer=m.moe_layers[at], gain=m.gain_handles[at],
                 attn=attention_weights()[int(rng.integers(ATTN_SETS))], cos=m.cos, sin=m.sin, x=_rows(tokens, D, gen),
                 k=cache(HKV, start + tokens, HD), v=cache(HKV, start + tokens, HD))
    elif kind == "moe_host":
        m = moe_model()
        at = int(rng.integers(BLOCKS))
        s.update(layer=m.moe_layers[at].handle, gain=m.gain_handles[at], x=_rows(case["tokens"], D, gen).cpu().numpy())
    elif kind == "qkv_host":
        s.update(attn=attention_weights()[int(rng.integers(ATTN_SETS))], x=_rows(case["tokens"], D, gen).cpu().numpy())
    elif kind == "q1_decode":
        s["decoder"], s["context"] = q1_decoder(), case["context"]
        s["decoder"].set_position(case["context"])
        s["decoder"].capture(case["context"])
        s["token"], s["next"] = _pinned_token(int(rng.integers(VOCAB))), _pinned_token(0)
    elif kind == "q1_prefill":
        w, g = q1_host_model()
        s.update(w=w, g=g, dims=(case["tokens"], Q_D, Q_HOST_BLOCKS, Q_H, Q_HKV, Q_HD, Q_FFN), export=case["export"],
                 x=np.rint(rng.standard_normal((case["tokens"], Q_D)) * 0.05 * (1 << FRAC)).astype(np.int64))
    elif kind == "q1_step":
        w, g = q1_host_model()
        B, context = case["sequences"], case["context"]
        ctx = q1_gpu.decode_ctx_create((B, Q_HOST_BLOCKS, Q_H, Q_HKV, Q_HD, Q_D, Q_FFN, VOCAB), w, g, FRAC, 1, _q1_inv_sqrt(), 320)
        weakref.finalize(s, q1_gpu.decode_ctx_free, ctx)
        s["positions"] = np.array([context - (b * 7) % 24 for b in range(B)], np.int64)      # sequences that began at other times
        for b in range(B):
            shape = (Q_HOST_BLOCKS, Q_HKV, int(s["positions"][b]), Q_HD)
            q1_gpu.decode_ctx_seed_seq(ctx, b, rng.integers(-(1 << 17), 1 << 17, size=shape), rng.integers(-(1 << 17), 1 << 17, size=shape))
        s.update(ctx=ctx, x=np.rint(rng.standard_normal((B, Q_D)) * 0.05 * (1 << FRAC)).astype(np.int64))
    else:
        raise ValueError(f"unknown case {case}")
    return s


def _q1_inv_sqrt():
    return int(round((1.0 / Q_HD ** 0.5) * (1 << FRAC)))


# --------------------------------------------------------------------------------------------------------------- a pass ---
def run(s):
    kind = s["kind"]
    if kind in ("decode", "q1_decode"):
        dec = s["decoder"]
        dec.set_position(s["context"])
        dec.decode_token(s["token"], s["next"])
        last = dec.attn[-1] if kind == "decode" else dec.layers[-1]
        return {"next": s["next"], "logits": dec.logits, "x": dec.x, "k": last["k"], "v": last["v"]}
    if kind == "step":
        dec = s["decoder"]
        dec.tokens.copy_(s["tokens"])
        dec.step()
        return {"next": dec.tokens, "logits": dec.logits, "x": dec.x}
    if kind == "prefill":
        a, x = s["attn"], s["x"]
        h = device.rmsnorm(x, s["gain"], FA, 1)
        qkv = device.apply(a["wqkv"], h, QD + 2 * KD, FW)
        att = device.attention_prefill(qkv[:, :QD].contiguous(), qkv[:, QD:QD + KD].contiguous(), qkv[:, QD + KD:].contiguous(),
                                       s["k"], s["v"], s["start"], H, HKV, HD, FA, WINDOW if s["rope"] else 0, s["cos"], s["sin"], s["rope"])
        ao = device.apply(a["wo"], att, D, FW)
        moe, ids, gates = s["layer"].forward(h, FA, FW)
        return {"x": x + ao + moe, "ids": ids, "gates": gates, "k": s["k"], "v": s["v"]}
    if kind == "moe_host":
        return qk_cuda.moe_block(s["layer"], s["x"], TOP_K, FA, FW, s["gain"])
    if kind == "qkv_host":
        a = s["attn"]
        return qk_cuda.apply_resident_grouped((a["wq"], a["wk"], a["wv"]), s["x"], (QD, KD, KD), FW,
                                              (qk_cuda.PROFILE_Q, qk_cuda.PROFILE_K, qk_cuda.PROFILE_V))
    if kind == "q1_prefill":
        return q1_gpu.prefill_forward_gpu(s["x"], s["dims"], s["w"], s["g"], FRAC, 1, _q1_inv_sqrt(), export_kv=s["export"])
    return q1_gpu.decode_step(s["ctx"], s["x"], s["positions"], VOCAB)


# ------------------------------------------------------------------------------------------------------- work, tolerance ---
def _moe_work(tokens):
    """Router and expert products of one block: every expert that some row selects is read once."""
    expert = 2 * EFF * NB * 144 + D * (EFF // 256) * 210
    touched = EXPERTS * (1.0 - (1.0 - TOP_K / EXPERTS) ** tokens)
    return EXPERTS * NB * 144 + touched * expert + 16 * tokens * D, 2.0 * tokens * (EXPERTS * D + TOP_K * 3 * D * EFF)


def _attn_work(tokens, start, heads, kv_heads):
    """Visible K and V rows once, the products of every query with the keys it sees."""
    pairs = tokens * start + tokens * (tokens + 1) / 2.0
    return 2 * kv_heads * (start + tokens) * HD * 4, 4.0 * pairs * heads * HD


def _linears_work(tokens):
    weights = (QD + 2 * KD) * NB * 144 + D * (QD // 256) * 144
    return weights, 2.0 * tokens * D * (2 * QD + 2 * KD)


def _block_work(tokens, start):
    parts = [_moe_work(tokens), _attn_work(tokens, start, H, HKV), _linears_work(tokens)]
    return sum(p[0] for p in parts), sum(p[1] for p in parts)


def _q1_block_work(tokens, start):
    macs = Q_D * (2 * Q_H + 2 * Q_HKV) * Q_HD + 3 * Q_D * Q_FFN
    b, f = _attn_work(tokens, start, Q_H, Q_HKV)
    return macs // 128 * 20 + b, 2.0 * tokens * macs + f


def work(case):
    kind = case["kind"]
    head, q1_head = VOCAB * NB * 210, VOCAB * (Q_D // 128) * 20
    if kind == "decode":
        b, f = _block_work(1, case["context"])
        return {"bytes": BLOCKS * b + head + 8 * VOCAB, "flops": BLOCKS * f + 2.0 * VOCAB * D}
    if kind == "step":
        n = case["sequences"]
        (mb, mf), (lb, lf), (ab, af) = _moe_work(n), _linears_work(n), _attn_work(1, case["context"], H, HKV)
        return {"bytes": STEP_BLOCKS * (mb + lb + n * ab) + head + 8 * n * VOCAB, "flops": STEP_BLOCKS * (mf + lf + n * af) + 2.0 * n * VOCAB * D}
    if kind == "prefill":
        b, f = _block_work(case["tokens"], case["start"])
        return {"bytes": b, "flops": f}
    if kind == "moe_host":
        b, f = _moe_work(case["tokens"])
        return {"bytes": b, "flops": f}
    if kind == "qkv_host":
        return {"bytes": (QD + 2 * KD) * NB * 144 + 8 * case["tokens"] * (D + QD + 2 * KD), "flops": 2.0 * case["tokens"] * D * (QD + 2 * KD)}
    if kind == "q1_decode":
        b, f = _q1_block_work(1, case["context"])
        return {"bytes": Q_BLOCKS * b + q1_head + 8 * VOCAB, "flops": Q_BLOCKS * f + 2.0 * VOCAB * Q_D}
    if kind == "q1_prefill":
        b, f = _q1_block_work(case["tokens"], 0)
        return {"bytes": Q_HOST_BLOCKS * b + q1_head + 8 * case["tokens"] * Q_D, "flops": Q_HOST_BLOCKS * f + 2.0 * VOCAB * Q_D}
    n = case["sequences"]
    (wb, wf), (ab, af) = _q1_block_work(n, 0), _attn_work(1, case["context"], Q_H, Q_HKV)
    return {"bytes": Q_HOST_BLOCKS * (wb + n * ab) + q1_head + 8 * n * (Q_D + VOCAB), "flops": Q_HOST_BLOCKS * (wf + n * af) + 2.0 * n * VOCAB * Q_D}


def tolerance(case):
    return "exact"
