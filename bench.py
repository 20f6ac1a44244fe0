"""Benchmark of the integer decode path on B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference] [--workload decode|prefill|ep_decode|q1|q1_token]

Default workload, one step = one greedily decoded token of the synthetic 30B-A3B-shaped model at context 4096:
embedding row -> 48 blocks (RMSNorm, Q/K/V products, RoPE on sliding-window blocks, KV-cache append, exact
integer softmax attention, O product, MoE block: router, top-8 + sigmoid gates, gate/up with fused integer SiLU,
down with fused gate-weighted combine; x += attention + moe) -> output norm -> tied head over 151936 tokens ->
arg-max.  Weights are seeded synthetic blocks generated on the device; the KV cache is filled with seeded int32
values in place of a prefill.  A step streams 1.9 GB of distinct weights and 0.8 GB of cache, far above the
126 MB L2.

Printed JSON line (rank 0): `value` = tokens/s of the device-resident greedy chain (token id and position stay in
device cells; one CUDA-graph replay per token); `e2e` = the same through the public per-token call with the
token id going in and coming out through pinned host buffers; `e2e_abi` = the reference-facing host-buffer entries
(`qk_moe_ffn_batched`, `iie_moe_block_host`) on the config-1 block with NumPy buffers, host<->device copies inside the
timed call, next to the reference project's own CUDA producer called through the reference's own bridge;
`roofline` = the MoE gate/up kernel (largest single consumer of the step) timed alone with CUDA events against the
measured HBM copy bandwidth; `int8_peak` = an int8 GEMM (torch._int_mm, 8192^3) measured in the same run, the
denominator of the prefill line; `cpu_baseline` = the CPU oracle on this box's host cores for a bounded sample;
`config.moe_blocks_only` = the 48 MoE blocks alone.  Before timing, every stage of a token (embedding, norms,
projections, cache row, attention, MoE routing and output of every block, head logits, pick) is compared byte for
byte with the CPU oracle for four consecutive greedy tokens (all blocks of the first, a sample of the others), and
the replayed graph is compared with that oracle-checked chain.

`--impl reference` times the reference project's compiled CPU kernel (oracle/_ref) composed the way its engine
composes a decode step on the CPU: every step runs all the blocks and the head (two synthetic blocks' weights are
cycled through, so the kernel calls and their sizes are those of the whole model).
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

FA, FW = 16, 24
SUSTAIN_STEPS = 60         # replays before and after the timed steps, inside the clock sampler's window
D_MODEL, E_FFN, N_EXPERTS, TOP_K = 2048, 768, 128, 8
N_HEADS, N_KV, HEAD_DIM, VOCAB, WINDOW = 32, 4, 128, 151936, 4096


def ncu_figure(name: str):
    """A figure read off an ncu capture, kept as `key=value` lines in profiles/ncu_figures.txt; None when absent."""
    f = ROOT / "profiles" / "ncu_figures.txt"
    if f.exists():
        for line in f.read_text().splitlines():
            key, _, val = line.partition("=")
            if key.strip() == name:
                return float(val.split("#")[0])
    return None

WORKLOAD = ("config2_decode: batch-1 KV-cached greedy decode of the 30B-A3B-shaped model, 48 blocks (RMSNorm, Q/K/V, RoPE on "
            "sliding-window blocks, int32 KV cache at context 4096, exact integer softmax attention, O, MoE with 128 experts "
            "top-8 eff 768), tied Q6_K head over 151936 tokens, arg-max; Q4_K weights, Q6_K down and head")


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=32)
    ap.add_argument("--warmup", type=int, default=4)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--layers", type=int, default=48)
    ap.add_argument("--verify-layers", type=int, default=48, help="blocks checked against the CPU oracle before timing")
    ap.add_argument("--cpu-sample-layers", type=int, default=2)
    ap.add_argument("--context", type=int, default=4096, help="KV-cache rows already filled when decoding starts")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--workload", default="decode", choices=["decode", "prefill", "ep_decode", "q1", "q1_token", "q1_prefill"],
                    help="decode = the headline line (batch-1 MoE decode); the others print a line of the same "
                         "shape for the prefill, expert-parallel and Q1_0 configurations")
    ap.add_argument("--tokens", type=int, default=0, help="prefill: tokens per step (2048); ep_decode: sequences (64)")
    return ap.parse_args()


# ------------------------------------------------------------------------------------------------ clocks ---
class ClockSampler:
    """Samples nvidia-smi clocks and throttle reasons while a timed region runs."""
    FIELDS = ("clocks.sm,clocks.max.sm,clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index, self.proc, self.lines = index, None, []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.FIELDS}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except OSError:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *exc):
        if self.proc:
            time.sleep(0.15)
            self.proc.terminate()
            try:
                self.proc.wait(timeout=2)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self) -> dict:
        sm, mx, reasons = [], 0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            parts = [p.strip() for p in ln.split(",")]
            if len(parts) < 6:
                continue
            try:
                sm.append(float(parts[0])); mx = max(mx, float(parts[1]))
            except ValueError:
                continue
            for name, val in zip(names, parts[2:6]):
                if val.lower().startswith("active"):
                    reasons.add(name)
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": mx or None, "reasons": sorted(reasons),
                "samples": len(sm)}


def measured_peak_gbs():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        return float(json.loads(p.read_text())["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


# -------------------------------------------------------------------------------------- reference arm -----
def host_cores() -> int:
    try:
        return len(os.sched_getaffinity(0))
    except AttributeError:
        return os.cpu_count() or 1


def use_all_host_threads() -> int:
    """The CPU checkers are OpenMP code; a launcher may have exported OMP_NUM_THREADS=1 for its workers (torchrun does).
    Give the OpenMP runtime they bind every core this process may use and return that count."""
    import ctypes
    n = host_cores()
    os.environ["OMP_NUM_THREADS"] = str(n)
    try:
        ctypes.CDLL("libgomp.so.1", mode=ctypes.RTLD_GLOBAL).omp_set_num_threads(n)
    except (OSError, AttributeError):
        pass
    return n


class CpuDecodeStep:
    """One decode step on the CPU, composed as the reference's engine composes it on its CPU path
    (north-mini-code/src/nmc/engine.py:429-443 for the experts, cohere2.py:357-376 for the block, :201-204 for the head):
    per block the four attention projections, NumPy integer attention over `context` cached keys, router, top-k, the
    routed experts' gate / up / down products with integer SiLU and the gate-weighted sum; then the tied head.
    `n_sets` synthetic blocks are built and cycled through, so a step of `layers` blocks makes the kernel calls of the
    whole model without holding 19 GB of host weights.  kind "reference": products by the reference project's compiled
    kernel (oracle/_ref); "port": this repository's C oracle."""

    def __init__(self, kind: str, n_sets: int, context: int, seed: int = 1):
        from oracle import native as onat
        from oracle import qk_oracle as o
        self.o, self.onat, self.kind, self.context = o, onat, kind, context
        self.lin = onat.ref_qk_linear if kind == "reference" else onat.qk_linear
        rng = np.random.default_rng(seed)
        nb = D_MODEL // 256
        self.sets = []
        for li in range(n_sets):
            router, gate, up, down, _ = o.synth_moe(seed * 1000 + li, D_MODEL, E_FFN, N_EXPERTS, 1, FA)
            self.sets.append({
                "wq": o.synth_q4k(rng, N_HEADS * HEAD_DIM, nb), "wk": o.synth_q4k(rng, N_KV * HEAD_DIM, nb),
                "wv": o.synth_q4k(rng, N_KV * HEAD_DIM, nb), "wo": o.synth_q4k(rng, D_MODEL, N_HEADS * HEAD_DIM // 256),
                "router": router, "gate": gate, "up": up, "down": down,
                "gain": o.to_fixed(np.abs(rng.standard_normal(D_MODEL)) + 0.5, FA),
                "k": rng.integers(-(1 << 18), 1 << 18, size=(N_KV, context + 1, HEAD_DIM), dtype=np.int64),
                "v": rng.integers(-(1 << 18), 1 << 18, size=(N_KV, context + 1, HEAD_DIM), dtype=np.int64)})
        self.embd = o.synth_q6k(rng, VOCAB, nb)
        self.out_gain = o.to_fixed(np.abs(rng.standard_normal(D_MODEL)) + 0.5, FA)
        self.cos, self.sin = o.build_rope_tables(1, HEAD_DIM, 50000.0, FA)
        self.x0 = o.to_fixed(rng.standard_normal((1, D_MODEL)), FA)

    def block(self, x, W, full: bool):
        o, lin, nb, ctx = self.o, self.lin, D_MODEL // 256, self.context
        h = o.rmsnorm_fixed(x, FA, 1, W["gain"])
        q = lin(W["wq"], h, N_HEADS * HEAD_DIM, nb, FW, o.Q4_K).reshape(1, N_HEADS, HEAD_DIM)
        k = lin(W["wk"], h, N_KV * HEAD_DIM, nb, FW, o.Q4_K).reshape(1, N_KV, HEAD_DIM)
        v = lin(W["wv"], h, N_KV * HEAD_DIM, nb, FW, o.Q4_K).reshape(1, N_KV, HEAD_DIM)
        if not full:
            rot = lambda t: o.rope_fixed(np.transpose(t, (1, 0, 2)), self.cos, self.sin, FA).transpose(1, 0, 2)
            q, k = rot(q), rot(k)
        W["k"][:, ctx] = k[0]; W["v"][:, ctx] = v[0]
        att = o.attention_cached(q, W["k"], W["v"], ctx, N_HEADS, N_KV, FA, None if full else WINDOW)
        ao = lin(W["wo"], att, D_MODEL, N_HEADS * HEAD_DIM // 256, FW, o.Q4_K)
        logits = lin(W["router"], h, N_EXPERTS, nb, FW, o.Q4_K)[0]
        sel = o.topk_lowidx(logits, TOP_K)
        gates = o.sigmoid_fixed(logits[sel], FA)
        moe = np.zeros(D_MODEL, dtype=object)
        for j, e in enumerate(sel):
            g = o.silu_int(lin(W["gate"][e], h, E_FFN, nb, FW, o.Q4_K), FA)
            u = lin(W["up"][e], h, E_FFN, nb, FW, o.Q4_K)
            dn = lin(W["down"][e], o.mul_shift(g, u, FA), D_MODEL, E_FFN // 256, FW, o.Q6_K)[0].astype(object)
            moe += (dn * int(gates[j])) >> FA
        return x + ao + moe.astype(np.int64)

    def step(self, layers: int) -> int:
        o = self.o
        x = self.x0
        for li in range(layers):
            x = self.block(x, self.sets[li % len(self.sets)], li % 4 == 0)
        hn = o.rmsnorm_fixed(x, FA, 1, self.out_gain)
        logits = self.lin(self.embd, hn, VOCAB, D_MODEL // 256, FW, o.Q6_K)[0]
        return int(np.flatnonzero(logits == logits.max())[0])


def run_reference(args):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    use_all_host_threads()
    from oracle import native as onat
    kind = "reference" if onat.ref_available() else "port"
    cpu = CpuDecodeStep(kind, 2, args.context)
    for _ in range(args.warmup):
        cpu.step(args.layers)
    times = []
    t_all = time.perf_counter()
    for _ in range(args.steps):
        t0 = time.perf_counter()
        cpu.step(args.layers)
        times.append(time.perf_counter() - t0)
    wall = time.perf_counter() - t_all
    step_s = wall / max(args.steps, 1)
    value = 1.0 / step_s
    sample = (f"every step: {args.layers} blocks (4 projections, attention over {args.context} keys, router, top-{TOP_K}, "
              f"{TOP_K} experts) and the head over {VOCAB} tokens; weights of 2 synthetic blocks cycled")
    print(json.dumps({
        "impl": "reference", "metric": "decode_tok_per_s", "value": value, "unit": "tok/s", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": step_s * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "int64", "data": "synthetic",
        "config": {"workload": WORKLOAD, "layers": args.layers, "context": args.context, "l2": "n/a (CPU)"},
        "cpu_baseline": {"value": value, "unit": "tok/s", "cores": host_cores(), "kind": kind, "sample": sample},
        "e2e": {"value": value, "unit": "tok/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "wall_s": wall, "ms_per_step_median": float(np.median(times)) * 1e3,
    }))


def int8_peak():
    """int8 x int8 -> int32 GEMM throughput of this GPU, measured in this run (torch._int_mm, 8192^3, 2*N^3 integer
    operations): best of 10 launches (burst) and back to back for ~2 s (sustained).  The denominator of the prefill line."""
    import torch
    n = 8192
    a = torch.randint(-128, 127, (n, n), dtype=torch.int8, device="cuda")
    b = torch.randint(-128, 127, (n, n), dtype=torch.int8, device="cuda")
    ops = 2.0 * n ** 3
    for _ in range(3):
        torch._int_mm(a, b)
    torch.cuda.synchronize()
    best = float("inf")
    for _ in range(10):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(); torch._int_mm(a, b); e1.record(); torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1))
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    reps = max(20, int(2000.0 / best))
    e0.record()
    for _ in range(reps):
        torch._int_mm(a, b)
    e1.record(); torch.cuda.synchronize()
    sustained_ms = e0.elapsed_time(e1) / reps
    del a, b
    return {"burst_tops": ops / (best * 1e-3) / 1e12, "sustained_tops": ops / (sustained_ms * 1e-3) / 1e12,
            "how": "torch._int_mm 8192^3 int8, 2*N^3 ops; best of 10 and mean of a ~2 s loop, CUDA events"}


_BRIDGE_PROBE = r'''
import json, sys, time
import numpy as np
sys.path.insert(0, sys.argv[1])                       # the repository root: oracle generators only
from oracle import qk_oracle as o
from nmc import qk_cuda as q                          # the reference's own bridge (baseline/_ref), library from BONSAI_BIN_DIR
assert q.available(), "bridge reports the library unusable"
FA, FW, d, eff, E, k, T = 16, 24, 2048, 768, 128, 8, 16
router, gate, up, down, h = o.synth_moe(0, d, eff, E, T)
sel = np.load(sys.argv[2])["config1_ids"]; want = np.load(sys.argv[2])["config1_out"]
logits = o.qk_linear(router, h, E, d // 256, FW, o.Q4_K)
gates = np.stack([o.sigmoid_fixed(logits[t][sel[t]], FA) for t in range(T)])
need = sorted(set(int(e) for e in sel.reshape(-1)))
gh = {e: q.register_weight(gate[e], eff, d // 256, q.Q4_K) for e in need}
uh = {e: q.register_weight(up[e], eff, d // 256, q.Q4_K) for e in need}
dh = {e: q.register_weight(down[e], d, eff // 256, q.Q6_K) for e in need}
flat = lambda hs: [hs[int(e)] for t in range(T) for e in sel[t]]
G, U, D = flat(gh), flat(uh), flat(dh)
out = q.moe_ffn_batched(G, U, D, T, k, h, gates.reshape(-1), d, eff, FA, FW)
assert out is not None and np.array_equal(out, want), "bytes differ from the golden block output"
reps = int(sys.argv[3])
ts = []
for _ in range(reps):
    t0 = time.perf_counter(); q.moe_ffn_batched(G, U, D, T, k, h, gates.reshape(-1), d, eff, FA, FW); ts.append(time.perf_counter() - t0)
print(json.dumps({"ms_per_call": float(np.median(ts)) * 1e3, "calls": reps, "library": str(q._so_path())}))
'''


def reference_bridge_timing(lib_dir: Path, reps: int = 20):
    """`qk_moe_ffn_batched` on the config-1 block (16 tokens, 128 experts, top-8) called through the REFERENCE's own bridge
    module, with `lib_dir/libnmc_qk_cuda.so` as the library it loads: once for the reference's CUDA producer built for
    sm_100a (baseline/_ref/bin), once for this repository's library.  A child process each, because the bridge binds one
    library per process.  Returns a dict, or {"unavailable": why}."""
    ref = ROOT / "baseline" / "_ref" / "north-mini-code"
    if not (ref / "src" / "nmc" / "qk_cuda.py").exists() or not (lib_dir / "libnmc_qk_cuda.so").exists():
        return {"unavailable": "reference bridge or library not installed under baseline/_ref"}
    env = dict(os.environ)
    env["BONSAI_BIN_DIR"] = str(lib_dir)
    env["PYTHONPATH"] = str(ref / "src")
    env.pop("BONSAI_NOTARY_HOME", None)
    try:
        run = subprocess.run([sys.executable, "-c", _BRIDGE_PROBE, str(ROOT), str(ROOT / "tests" / "golden" / "moe.npz"), str(reps)],
                             env=env, capture_output=True, text=True, timeout=600)
    except subprocess.TimeoutExpired:
        return {"unavailable": "timed out"}
    if run.returncode != 0:
        return {"unavailable": (run.stderr.strip().splitlines() or ["failed"])[-1][:200]}
    return json.loads(run.stdout.strip().splitlines()[-1])


def e2e_abi(reps: int = 20):
    """The reference-facing entries with HOST buffers on the config-1 block (seed 0, 16 tokens, 128 experts, top-8):
    `qk_moe_ffn_batched` (what Engine._moe calls) and `iie_moe_block_host` (routing included), wall clock around the
    call, uploads and downloads inside it; results compared with the golden bytes first."""
    from integer_inference_engine_b200 import device, qk_cuda
    from oracle import qk_oracle as o
    d, eff, E, k, T = D_MODEL, E_FFN, N_EXPERTS, TOP_K, 16
    g = np.load(ROOT / "tests" / "golden" / "moe.npz")
    router, gate, up, down, h = o.synth_moe(0, d, eff, E, T)
    sel = g["config1_ids"]
    logits = o.qk_linear(router, h, E, d // 256, FW, o.Q4_K)
    gates = np.stack([o.sigmoid_fixed(logits[t][sel[t]], FA) for t in range(T)])
    rh = qk_cuda.register_weight(router, E, d // 256, o.Q4_K)
    gh = [qk_cuda.register_weight(w, eff, d // 256, o.Q4_K) for w in gate]
    uh = [qk_cuda.register_weight(w, eff, d // 256, o.Q4_K) for w in up]
    dh = [qk_cuda.register_weight(w, d, eff // 256, o.Q6_K) for w in down]
    layer = device.MoELayer(rh, gh, uh, dh, k, d, eff)
    flat = lambda hs: [hs[int(e)] for t in range(T) for e in sel[t]]
    G, U, Dn, gflat = flat(gh), flat(uh), flat(dh), gates.reshape(-1)
    out = {}
    a = qk_cuda.moe_ffn_batched(G, U, Dn, T, k, h, gflat, d, eff, FA, FW)
    b = qk_cuda.moe_block(layer.handle, h, k, FA, FW)
    assert a is not None and np.array_equal(a, g["config1_out"]), "qk_moe_ffn_batched differs from the golden block output"
    assert b is not None and np.array_equal(b[0], g["config1_out"]) and np.array_equal(b[1], sel), "iie_moe_block_host differs"
    for name, fn in (("qk_moe_ffn_batched", lambda: qk_cuda.moe_ffn_batched(G, U, Dn, T, k, h, gflat, d, eff, FA, FW)),
                     ("iie_moe_block_host", lambda: qk_cuda.moe_block(layer.handle, h, k, FA, FW))):
        ts = []
        for _ in range(reps):
            t0 = time.perf_counter(); fn(); ts.append(time.perf_counter() - t0)
        ms = float(np.median(ts)) * 1e3
        routed = name == "iie_moe_block_host"
        out[name] = {"ms_per_call": ms, "tok_per_s": T / (ms * 1e-3), "tokens": T,
                     "h2d_bytes_per_call": h.nbytes + (0 if routed else gflat.nbytes + 3 * len(G) * 8),
                     "d2h_bytes_per_call": h.nbytes + (T * k * 12 if routed else 0)}
    layer.close()
    return out


# ---------------------------------------------------------------------------------------------- our arm ---
def check_moe_block(stack, li, hn, ids, gates, out):
    """One block's routing and output against the C oracle, using the weights exported back from the device."""
    from integer_inference_engine_b200 import device
    from oracle import native as onat
    from oracle import qk_oracle as o
    nb_in, nb_dn = D_MODEL // 256, E_FFN // 256
    hs = stack.handles[li]
    router = device.export_weight(hs["router"], N_EXPERTS, nb_in, o.Q4_K)
    logits = onat.qk_linear(router, hn, N_EXPERTS, nb_in, FW, o.Q4_K)
    sel = np.stack([onat.topk_lowidx(r, TOP_K) for r in logits])
    assert np.array_equal(ids, sel), f"block {li}: router ids"
    gref = np.stack([onat.sigmoid(logits[t][sel[t]], FA) for t in range(sel.shape[0])])
    assert np.array_equal(gates, gref), f"block {li}: gates"
    ref = np.zeros((hn.shape[0], D_MODEL), dtype=object)
    for t in range(hn.shape[0]):
        for j, e in enumerate(sel[t]):
            gw = device.export_weight(hs["gate"][e], E_FFN, nb_in, o.Q4_K)
            uw = device.export_weight(hs["up"][e], E_FFN, nb_in, o.Q4_K)
            dw = device.export_weight(hs["down"][e], D_MODEL, nb_dn, o.Q6_K)
            g = onat.silu(onat.qk_linear(gw, hn[t:t + 1], E_FFN, nb_in, FW, o.Q4_K), FA)
            u = onat.qk_linear(uw, hn[t:t + 1], E_FFN, nb_in, FW, o.Q4_K)
            dn = onat.qk_linear(dw, o.mul_shift(g, u, FA), D_MODEL, nb_dn, FW, o.Q6_K)[0].astype(object)
            ref[t] += (dn * int(gref[t, j])) >> FA
    assert np.array_equal(out, ref.astype(np.int64)), f"block {li}: block output"


def verify_token(model, token: int, n_check: int, check_blocks=None):
    """Eager walk of one decode step at the model's current position; every stage of the first `n_check` blocks (or of the
    blocks listed in `check_blocks`), the head and the pick are compared with the CPU oracle fed with the SAME stage inputs
    (exported weights, host copies of the caches).  Leaves the appended cache rows in place and returns the pick."""
    import torch

    from integer_inference_engine_b200 import device
    from oracle import native as onat
    from oracle import qk_oracle as o
    d, H, Hkv, hd, nb = model.d, model.H, model.Hkv, model.hd, model.d // 256
    pos = int(model.pos.item())
    cos, sin = model.cos[pos:pos + 1].cpu().numpy(), model.sin[pos:pos + 1].cpu().numpy()
    do_head = n_check > 0 or bool(check_blocks)
    embd_raw = device.export_weight(model.embd, model.vocab, nb, o.Q6_K) if do_head else None
    x = device.embed(model.embd, token, d, FA)
    if do_head:
        row = embd_raw[token * nb * 210:(token + 1) * nb * 210]
        assert np.array_equal(x.cpu().numpy()[0], o.dequant(row, 1, nb, o.Q6_K, FA)[0]), "embedding row"
    checked = 0
    for li in range(model.n_layers):
        a, gain_h = model.attn[li], model.moe.gains[li]
        full = model.layer_is_full(li)
        h = device.rmsnorm(x, gain_h, FA, 1)
        qr, kr = H * hd, Hkv * hd
        qkv = device.apply(a["wqkv"], h, qr + 2 * kr, FW)
        q_in, k, v = qkv[:, :qr].contiguous(), qkv[:, qr:qr + kr].contiguous(), qkv[:, qr + kr:].contiguous()
        att = device.attention_decode(q_in.view(-1), k.view(-1), v.view(-1), a["k"], a["v"], pos, H, Hkv, hd, FA,
                                      0 if full else model.window, model.cos, model.sin, 0 if full else 1).view(1, -1)
        ao = device.apply(a["wo"], att, d, FW)
        out, ids, gates = model.moe.layers[li].forward(h, FA, FW)
        # the two block entries the timed step uses (MoE half, then attention half) on a copy of the row
        xb = x.clone()
        model.moe.layers[li].block(xb, gain_h, FA, FW, 1, out=xb, want_routes=False)
        device.attention_block(a["wqkv"], a["wo"], xb, a["k"], a["v"], pos, H, Hkv, hd, FA, FW, 0 if full else model.window,
                               model.cos, model.sin, 0 if full else 1)
        torch.cuda.synchronize()
        assert device.read_flags() == 0, f"block {li}: envelope flag raised"
        assert torch.equal(xb, x + ao + out), f"block {li}: block entries differ from the stage-by-stage composition"
        if li < n_check or (check_blocks is not None and li in check_blocks):
            xn, hn = x.cpu().numpy(), h.cpu().numpy()
            assert np.array_equal(hn, o.rmsnorm_fixed(xn, FA, 1, model.moe.handles[li]["gain"].cpu().numpy())), f"block {li}: RMSNorm"
            w = device.export_weight(a["wqkv"], qr + 2 * kr, nb, o.Q4_K)
            assert np.array_equal(qkv.cpu().numpy(), onat.qk_linear(w, hn, qr + 2 * kr, nb, FW, o.Q4_K)), f"block {li}: fused QKV"
            qn, kn = q_in.cpu().numpy().reshape(1, H, hd), k.cpu().numpy().reshape(1, Hkv, hd)
            if not full:
                rot = lambda t: o.rope_fixed(np.transpose(t, (1, 0, 2)), cos, sin, FA).transpose(1, 0, 2)
                qn, kn = rot(qn), rot(kn)
            lo = 0 if full else max(0, pos - model.window + 1)
            ck = a["k"][:, :pos + 1].cpu().numpy().astype(np.int64); cv = a["v"][:, :pos + 1].cpu().numpy().astype(np.int64)
            assert np.array_equal(ck[:, pos], kn[0]) and np.array_equal(cv[:, pos], v.cpu().numpy().reshape(Hkv, hd)), f"block {li}: cache row"
            want = o.attention_cached(qn, ck, cv, pos, H, Hkv, FA, None if full else model.window)
            assert np.array_equal(att.cpu().numpy(), want), f"block {li}: attention (keys {lo}..{pos})"
            wo = device.export_weight(a["wo"], d, H * hd // 256, o.Q4_K)
            assert np.array_equal(ao.cpu().numpy(), onat.qk_linear(wo, att.cpu().numpy(), d, H * hd // 256, FW, o.Q4_K)), f"block {li}: wo"
            check_moe_block(model.moe, li, hn, ids.cpu().numpy(), gates.cpu().numpy(), out.cpu().numpy())
            checked += 1
        x = x + ao + out
    hn = device.rmsnorm(x, model.out_gain_h, FA, 1)
    logits = device.apply(model.embd, hn, model.vocab, FW)
    tok = int(device.argmax(logits.view(-1)).item())
    if do_head:
        assert np.array_equal(hn.cpu().numpy(), o.rmsnorm_fixed(x.cpu().numpy(), FA, 1, model.out_gain.cpu().numpy())), "output norm"
        want = onat.qk_linear(embd_raw, hn.cpu().numpy(), model.vocab, nb, FW, o.Q6_K)[0]
        assert np.array_equal(logits.cpu().numpy()[0], want), "head logits"
        assert tok == int(np.flatnonzero(want == want.max())[0]), "greedy pick"
    return checked, tok


def run_ours(args):
    import torch
    import torch.distributed as dist

    from integer_inference_engine_b200 import device, qk_cuda
    from integer_inference_engine_b200.model import SyntheticDecoder

    rank, world = int(os.environ.get("RANK", "0")), int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    if world > 1:
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    if not qk_cuda.available():
        raise SystemExit("CUDA library or GPU missing: there is no fallback path")

    n_e2e = 0 if args.no_e2e else max(2, min(args.steps, 16))
    n_pad = 0 if args.no_e2e else 2 * SUSTAIN_STEPS               # identical replays around the timed region (clock sampling)
    total_steps = args.warmup + args.steps + n_e2e + n_pad + 24
    model = SyntheticDecoder(n_layers=args.layers, d_model=D_MODEL, n_heads=N_HEADS, n_kv=N_KV, head_dim=HEAD_DIM, e_ffn=E_FFN,
                             n_experts=N_EXPERTS, top_k=TOP_K, vocab=VOCAB, context=args.context, max_new=total_steps + 8,
                             window=WINDOW, seed=1 + rank, fa=FA, fw=FW)
    stack = model.moe
    first_token = 1234 + rank
    pos0 = model.context
    pos_bound = pos0 + total_steps

    # ---- parity before timing: four consecutive greedy tokens walked stage by stage against the CPU oracle (every block
    # of the first token, a spread of blocks of the others, head and pick of each), then the step entries and the replayed
    # graph must reproduce that oracle-checked chain --------------------------------------------------------------------
    n_chain = 4
    oracle_ids, checked, tok = [], 0, first_token
    for i in range(n_chain):
        model.set_position(pos0 + i)
        if rank == 0:
            blocks = None if i == 0 else set(range(i, args.layers, max(1, args.layers // 4)))
            n_chk, tok = verify_token(model, tok, args.verify_layers if i == 0 else 0, blocks if args.verify_layers else None)
        else:
            n_chk, tok = verify_token(model, tok, 0)
        checked += n_chk
        oracle_ids.append(tok)
    model.token.fill_(first_token); model.set_position(pos0)
    eager_ids = []
    for i in range(n_chain):
        model.step(pos0 + i)
        eager_ids.append(int(model.token.item()))
    assert eager_ids == oracle_ids, f"step entries {eager_ids} differ from the oracle-checked chain {oracle_ids}"
    model.token.fill_(first_token); model.set_position(pos0)
    l0 = device.launch_count()
    model.capture(pos_bound)
    launches_per_step = (device.launch_count() - l0) // 2         # capture() runs the step twice
    replay_ids = []
    for i in range(n_chain):
        model.replay()
        replay_ids.append(int(model.token.item()))
    assert replay_ids == oracle_ids, f"graph replay {replay_ids} differs from the oracle-checked chain {oracle_ids}"

    # ---- device-resident timing: the greedy chain continues, one graph replay per token ----------------------------
    for i in range(args.warmup):
        model.replay()
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with ClockSampler(local) as clk:
        # the timed K steps sit inside a longer run of identical replays, so that the 100 ms clock sampler sees the load
        for i in range(n_pad // 2):
            model.replay()
        ev0.record()
        for i in range(args.steps):
            model.replay()
        ev1.record()
        for i in range(n_pad // 2):
            model.replay()
        torch.cuda.synchronize()
    ms = ev0.elapsed_time(ev1)
    if world > 1:
        t = torch.tensor([ms], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    assert device.read_flags() == 0, "an activation left the exact envelope during the timed region"
    pos_timed = int(model.pos.item())

    # ---- the MoE blocks alone (the hot path of this build) and the roofline of its dominant kernel --------------------
    peak, peak_kind = measured_peak_gbs()
    rng = np.random.default_rng(1000 + rank)
    from oracle import qk_oracle as o
    table = torch.from_numpy(o.to_fixed(rng.standard_normal((4, D_MODEL)), FA)).cuda()
    side = torch.cuda.Stream()
    x_moe = table[:1].clone()
    stack.decode_step(x_moe.clone(), FW)
    torch.cuda.synchronize()
    g_moe = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        with torch.cuda.graph(g_moe, stream=side):
            stack.decode_step(x_moe, FW)
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    g_moe.replay(); torch.cuda.synchronize()
    e0.record()
    for _ in range(8):
        g_moe.replay()
    e1.record(); torch.cuda.synchronize()
    moe_only_ms = e0.elapsed_time(e1) / 8
    h_probe = device.rmsnorm(table[:1], stack.gains[0], FA, 1)
    outs = torch.zeros_like(h_probe)
    for layer in stack.layers:                                   # leaves ids/gates/limbs of the last block in place
        layer.forward(h_probe, FA, FW, out=outs, accumulate=True, want_routes=False)
    torch.cuda.synchronize()
    reps = 3

    def time_stage(mask):
        """Average device time of one stage over all blocks, captured as one graph and replayed."""
        x_probe = table[:1].clone()
        device.set_stage_mask(mask)
        g2 = torch.cuda.CUDAGraph()
        with torch.cuda.stream(side):
            with torch.cuda.graph(g2, stream=side):
                for layer, gain_h in zip(stack.layers, stack.gains):
                    layer.block(x_probe, gain_h, FA, FW, 1, out=outs, want_routes=False)
        device.set_stage_mask(0)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        g2.replay()
        torch.cuda.synchronize()
        e0.record()
        for _ in range(reps):
            g2.replay()
        e1.record()
        torch.cuda.synchronize()
        device.read_flags()
        return e0.elapsed_time(e1) / (reps * len(stack.layers))

    route_ms, gateup_ms, down_ms = time_stage(2), time_stage(8), time_stage(16)
    gateup_bytes = TOP_K * 2 * E_FFN * (D_MODEL // 256) * 144
    down_bytes = TOP_K * D_MODEL * (E_FFN // 256) * 210
    achieved = gateup_bytes / (gateup_ms * 1e-3) / 1e9

    # ---- end to end: the public per-token call, token id in and out through pinned host buffers -----------------------
    e2e = None
    if n_e2e:
        tok_in = torch.zeros(1, dtype=torch.int32).pin_memory()
        tok_out = torch.zeros(1, dtype=torch.int32).pin_memory()
        tok_in[0] = int(model.token.item())
        model.decode_token(tok_in, tok_out)                       # untimed first call
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for i in range(n_e2e):
            tok_in[0] = tok_out[0]
            model.decode_token(tok_in, tok_out)
        e2e_s = (time.perf_counter() - t0) / n_e2e
        if world > 1:
            t = torch.tensor([e2e_s], device="cuda")
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            e2e_s = float(t.item())
        e2e = {"value": world / e2e_s, "unit": "tok/s", "h2d_bytes_per_step": 4, "d2h_bytes_per_step": 4, "steps": n_e2e}
    assert device.read_flags() == 0

    # with more than one rank the path shards (experts over ranks, sequences over ranks): measure that step too
    ep_res = None
    w_bytes, kv_bytes, one_launch = model.weight_bytes_per_token(), model.kv_bytes_per_token(pos_timed), model.kernel is not None
    moe_weight_bytes = stack.weight_bytes_per_token()
    if world > 1 and not args.no_e2e:
        del model, stack
        qk_cuda.free_all()
        torch.cuda.empty_cache()
        ep_args = argparse.Namespace(**vars(args))
        ep_args.tokens = 64
        ep_res = ep_decode_measure(ep_args, rank, world, local, 10, 3)
    if rank != 0:
        if world > 1:
            dist.destroy_process_group()
        return
    abi, i8 = None, None
    if not args.no_e2e:
        i8 = int8_peak()
        # the reference's own CUDA producer first, in its own process, through the reference's own bridge; then this library
        # through the same bridge call, and through this repository's bridge
        abi = {"workload": "config1 block: 16 tokens, 128 experts, top-8, host NumPy buffers, copies inside the call",
               "reference_bridge_with_reference_cuda_producer": reference_bridge_timing(ROOT / "baseline" / "_ref" / "bin"),
               "reference_bridge_with_this_library": reference_bridge_timing(ROOT / "integer_inference_engine_b200" / "lib")}
        abi.update(e2e_abi())
    cpu = None
    if args.cpu_sample_layers > 0:
        n_cpu = min(args.cpu_sample_layers, args.layers)
        use_all_host_threads()
        step = CpuDecodeStep("port", n_cpu, args.context)
        step.step(n_cpu)                                       # warm-up
        t0 = time.perf_counter(); step.step(n_cpu); t_blocks_head = time.perf_counter() - t0
        t0 = time.perf_counter(); step.step(0); t_head = time.perf_counter() - t0
        per_block = (t_blocks_head - t_head) / n_cpu
        cpu = {"value": 1.0 / (per_block * args.layers + t_head), "unit": "tok/s", "cores": host_cores(), "kind": "port",
               "sample": f"{n_cpu} blocks (attention over {args.context} keys + MoE) and the head, 1 token, "
                         f"scaled to {args.layers} blocks"}
    ms_step = ms / args.steps
    print(json.dumps({
        "metric": "decode_tok_per_s", "value": world * 1e3 / ms_step, "unit": "tok/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_step, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "int64", "data": "synthetic",
        "config": {"workload": WORKLOAD, "layers": args.layers, "context": args.context, "parallelism": f"replicas x{world}",
                   "l2": "inputs larger than L2: each step streams %d MB of distinct weights and %d MB of KV cache"
                         % (w_bytes // 2**20, kv_bytes // 2**20),
                   "weight_bytes_per_token": w_bytes, "kv_bytes_per_token": kv_bytes,
                   "step_hbm_frac_of_%s_peak" % peak_kind: (w_bytes + kv_bytes) / (ms_step * 1e-3) / 1e9 / peak,
                   "moe_blocks_only": {"ms_per_token": moe_only_ms, "tok_per_s": 1e3 / moe_only_ms,
                                       "weight_bytes": moe_weight_bytes},
                   "ep_decode": ep_res, "oracle_checked_blocks": checked, "oracle_checked_tokens": n_chain, "one_launch_decode": one_launch, "kv_cache": "seeded int32 values stand in for the prefill"},
        "clocks": dict(clk.summary(), window="the timed steps plus %d identical replays before and after them" % (n_pad // 2)),
        "e2e": e2e, "e2e_abi": abi, "int8_peak": i8, "gpu_launches": int(launches_per_step * args.steps),
        "roofline": {"bound": "hbm", "kernel": "stream_kernel<Q4_K, GATEUP>", "achieved": achieved, "peak": peak,
                     "peak_kind": peak_kind, "unit": "GB/s", "frac": achieved / peak, "traffic": ncu_figure("stream_kernel_gateup.dram_bytes_per_launch"),
                     "traffic_source": "dram__bytes_read.sum + dram__bytes_write.sum of one launch in an ncu capture of this kernel",
                     "bytes_per_launch": gateup_bytes, "ms_per_launch": gateup_ms,
                     "other_kernels_us": {"route": route_ms * 1e3, "down": down_ms * 1e3,
                                          "down_frac": down_bytes / (down_ms * 1e-3) / 1e9 / peak}},
        "cpu_baseline": cpu,
    }))
    if world > 1:
        dist.destroy_process_group()


# ------------------------------------------------------------------------------- secondary workloads ------
def _dist_setup():
    import torch
    import torch.distributed as dist
    rank, world = int(os.environ.get("RANK", "0")), int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    if world > 1:
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    return rank, world, local


def _timed(fn, steps, warmup, world, local):
    """W warm-up calls, then K calls between CUDA events on the current stream; max over ranks (ms total)."""
    import torch
    import torch.distributed as dist
    for i in range(warmup):
        fn(i)
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with ClockSampler(local) as clk:
        e0.record()
        for i in range(steps):
            fn(warmup + i)
        e1.record()
        torch.cuda.synchronize()
    ms = e0.elapsed_time(e1)
    if world > 1:
        t = torch.tensor([ms], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    return ms, clk.summary()


def _oracle_rows(stack, li, h_rows):
    """CPU checker for a few rows of block `li` (rows are independent in the MoE block)."""
    from integer_inference_engine_b200 import device
    from oracle import native as onat
    from oracle import qk_oracle as o
    hs = stack.handles[li]
    nb_in, nb_dn = D_MODEL // 256, E_FFN // 256
    router = device.export_weight(hs["router"], N_EXPERTS, nb_in, o.Q4_K)
    logits = onat.qk_linear(router, h_rows, N_EXPERTS, nb_in, FW, o.Q4_K)
    sel = np.stack([onat.topk_lowidx(r, TOP_K) for r in logits])
    lo, hi = stack.expert_range
    ref = np.zeros(h_rows.shape, dtype=object)
    for t in range(h_rows.shape[0]):
        gts = onat.sigmoid(logits[t][sel[t]], FA)
        for j, e in enumerate(sel[t]):
            if not lo <= e < hi:
                continue
            gw = device.export_weight(hs["gate"][e - lo], E_FFN, nb_in, o.Q4_K)
            uw = device.export_weight(hs["up"][e - lo], E_FFN, nb_in, o.Q4_K)
            dw = device.export_weight(hs["down"][e - lo], D_MODEL, nb_dn, o.Q6_K)
            g = onat.silu(onat.qk_linear(gw, h_rows[t:t + 1], E_FFN, nb_in, FW, o.Q4_K), FA)
            u = onat.qk_linear(uw, h_rows[t:t + 1], E_FFN, nb_in, FW, o.Q4_K)
            dn = onat.qk_linear(dw, o.mul_shift(g, u, FA), D_MODEL, nb_dn, FW, o.Q6_K)[0].astype(object)
            ref[t] += (dn * int(gts[j])) >> FA
    return sel, ref.astype(np.int64)


def run_prefill(args):
    """Prefill configuration: `tokens` (2048) rows through every MoE block per step, each rank a replica."""
    import torch
    import torch.distributed as dist

    from integer_inference_engine_b200 import device
    from integer_inference_engine_b200.synth import SyntheticMoEStack
    from oracle import qk_oracle as o
    rank, world, local = _dist_setup()
    T = args.tokens or 2048
    stack = SyntheticMoEStack(args.layers, D_MODEL, E_FFN, N_EXPERTS, TOP_K, seed=1 + rank, fa=FA)
    x0 = torch.from_numpy(o.to_fixed(np.random.default_rng(7 + rank).standard_normal((T, D_MODEL)), FA)).cuda()
    h = device.rmsnorm(x0, stack.gains[0], FA, 1)
    out, ids, _ = stack.layers[0].forward(h, FA, FW)
    torch.cuda.synchronize()
    assert device.read_flags() == 0
    rows = [0, T // 3, T - 1]
    h_rows = h[rows].cpu().numpy()
    if rank == 0:
        use_all_host_threads()
    t0 = time.perf_counter()
    sel, ref = _oracle_rows(stack, 0, h_rows)
    cpu_s = time.perf_counter() - t0
    assert np.array_equal(ids[rows].cpu().numpy(), sel) and np.array_equal(out[rows].cpu().numpy(), ref), "block 0 differs from the oracle"
    x = x0.clone()
    l0 = device.launch_count()
    shapes0 = device.prefill_launch_counts()
    stack.decode_step(x, FW)
    launches = device.launch_count() - l0
    shapes = [b - a for a, b in zip(shapes0, device.prefill_launch_counts())]

    def step(i):
        x.copy_(x0)
        stack.decode_step(x, FW)
    ms, clocks = _timed(step, args.steps, args.warmup, world, local)
    assert device.read_flags() == 0
    # the attention sublayer of the same prefill (scores, exact softmax, probability-value sums of T tokens): checked on a
    # small case against the oracle, then timed alone at the model's shape
    rng = np.random.default_rng(3)
    sq, sk, sv = (rng.integers(-(1 << 18), 1 << 18, size=(9, w), dtype=np.int64) for w in (4 * 64, 2 * 64, 2 * 64))
    skc = torch.zeros((2, 12, 64), dtype=torch.int32, device="cuda"); svc = torch.zeros_like(skc)
    got = device.attention_prefill(torch.from_numpy(sq).cuda(), torch.from_numpy(sk).cuda(), torch.from_numpy(sv).cuda(), skc, svc,
                                   0, 4, 2, 64, FA, 5)
    want = o.attention_cached(sq.reshape(9, 4, 64), sk.reshape(9, 2, 64).transpose(1, 0, 2), sv.reshape(9, 2, 64).transpose(1, 0, 2),
                              0, 4, 2, FA, 5)
    assert np.array_equal(got.cpu().numpy(), want), "prefill attention differs from the oracle"
    g = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *sh: torch.randint(-(1 << 18), 1 << 18, sh, generator=g, device="cuda", dtype=torch.int64)
    aq, ak, av = rnd(T, N_HEADS * HEAD_DIM), rnd(T, N_KV * HEAD_DIM), rnd(T, N_KV * HEAD_DIM)
    akc = torch.zeros((N_KV, T, HEAD_DIM), dtype=torch.int32, device="cuda"); avc = torch.zeros_like(akc)
    aout = torch.empty((T, N_HEADS * HEAD_DIM), dtype=torch.int64, device="cuda")
    att_ms, _ = _timed(lambda i: device.attention_prefill(aq, ak, av, akc, avc, 0, N_HEADS, N_KV, HEAD_DIM, FA, WINDOW, out=aout),
                       3, 1, world, local)
    assert device.read_flags() == 0
    # the two dense products of the same block (fused Q/K/V and O) at T rows: Q4_K matrices on the tcgen05 LINEAR tiles
    from integer_inference_engine_b200.qk_cuda import Q4_K
    from integer_inference_engine_b200.synth import synth_q4k
    nbd, qkv_rows, qd = D_MODEL // 256, (N_HEADS + 2 * N_KV) * HEAD_DIM, N_HEADS * HEAD_DIM
    wqkv = device.register_weight(synth_q4k(qkv_rows * nbd, g).view(-1), qkv_rows, nbd, Q4_K)
    wo = device.register_weight(synth_q4k(D_MODEL * (qd // 256), g).view(-1), D_MODEL, qd // 256, Q4_K)
    lin_qkv = torch.empty((T, qkv_rows), dtype=torch.int64, device="cuda")
    lin_o = torch.empty((T, D_MODEL), dtype=torch.int64, device="cuda")
    att_in = rnd(T, qd)

    def linears(i):
        device.apply(wqkv, h, qkv_rows, FW, out=lin_qkv)
        device.apply(wo, att_in, D_MODEL, FW, out=lin_o)
    lin_ms, _ = _timed(linears, 3, 1, world, local)
    assert device.read_flags() == 0
    if rank == 0:
        ms_step = ms / args.steps
        i8 = int8_peak()
        # integer operations of one MoE block: algorithmic = 2 per multiply-add of the three expert products of every
        # (token, expert) pair; issued = the same times the digit pairs the tiles multiply (activation digits x weight digits)
        pair_macs = TOP_K * T * D_MODEL * E_FFN
        nl_gu = 3 if shapes[0] else 4
        nl_dn = 5 if shapes[2] else 6
        algorithmic = 2.0 * 3 * pair_macs
        issued = 2.0 * pair_macs * (2 * nl_gu * 2 + nl_dn * 2)
        blk_s = ms_step / args.layers * 1e-3
        roofline = {"bound": "tensor", "kernel": "tile_kernel gate/up + down of one MoE block (router, sort and digit planes included in the time)",
                    "unit": "TOP/s", "peak": i8["sustained_tops"], "peak_kind": "int8 GEMM measured in this run (torch._int_mm, sustained)",
                    "achieved": algorithmic / blk_s / 1e12, "frac": algorithmic / blk_s / 1e12 / i8["sustained_tops"],
                    "issued_achieved": issued / blk_s / 1e12, "issued_frac": issued / blk_s / 1e12 / i8["sustained_tops"],
                    "digits": {"gate_up": {"activation": nl_gu, "weight": 2}, "down": {"activation": nl_dn, "weight": 2}},
                    "tile_launches": shapes, "traffic": None}
        cpu = {"value": len(rows) / cpu_s / args.layers, "unit": "tok/s", "cores": host_cores(), "kind": "port",
               "sample": f"{len(rows)} rows through router, top-{TOP_K} and their {TOP_K} experts of one block on the CPU oracle, scaled to {args.layers} blocks (rows are independent)"}
        print(json.dumps({
            "metric": "prefill_tok_per_s", "value": world * T * 1e3 / ms_step, "unit": "tok/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_step, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "int64 via int8 digit planes (tcgen05 kind::i8)", "data": "synthetic",
            "config": {"workload": f"config3_moe_prefill: {T} tokens x {args.layers} MoE blocks, grouped expert GEMMs",
                       "ms_per_block": ms_step / args.layers, "attention_prefill_ms_per_block": att_ms / 3, "qkv_o_linears_ms_per_block": lin_ms / 3,
                       "whole_block_ms": ms_step / args.layers + att_ms / 3 + lin_ms / 3,
                       "parallelism": f"replicas x{world}",
                       "l2": "inputs larger than L2 (1.2 GB of expert weights per block)", "oracle_checked_rows": len(rows)},
            "clocks": clocks, "gpu_launches": int(launches * args.steps), "int8_peak": i8, "roofline": roofline, "cpu_baseline": cpu}))
    if world > 1:
        dist.destroy_process_group()


def ep_decode_measure(args, rank, world, local, steps, warmup):
    """Config 4: `tokens` (64) concurrent sequences at context `args.context`, whole decode step (every block with attention
    over each sequence's own cache and the expert-parallel MoE, head, greedy picks), sequences data-parallel and experts
    sharded over the ranks; the step is one replayed CUDA graph.  Block 0 is checked against the CPU oracle for one sequence
    per rank before timing.  Returns the figures of the line (max over ranks)."""
    import torch
    import torch.distributed as dist

    from integer_inference_engine_b200 import device
    from integer_inference_engine_b200.ep_model import ExpertParallelDecoder
    from oracle import native as onat
    from oracle import qk_oracle as o
    S = args.tokens or 64
    m = ExpertParallelDecoder(S, n_layers=args.layers, d_model=D_MODEL, n_heads=N_HEADS, n_kv=N_KV, head_dim=HEAD_DIM, e_ffn=E_FFN,
                              n_experts=N_EXPERTS, top_k=TOP_K, vocab=VOCAB, context=args.context, max_new=4, window=WINDOW, seed=1,
                              fa=FA, fw=FW)
    # ---- parity of block 0 for this rank's first sequence: attention against the NumPy checker, MoE rows against the C oracle
    x0 = torch.from_numpy(o.to_fixed(np.random.default_rng(50 + rank).standard_normal((m.B, D_MODEL)), FA)).cuda()
    pos, nb, a0_, hs = m.position, D_MODEL // 256, m.attn[0], m.stack.handles[0]
    qd, kd = N_HEADS * HEAD_DIM, N_KV * HEAD_DIM
    h = device.rmsnorm(x0, m.stack.gains[0], FA, 1)
    qkv = device.apply(a0_["wqkv"], h, qd + 2 * kd, FW)
    att = device.attention_decode_batch(qkv[:, :qd].contiguous(), qkv[:, qd:qd + kd].contiguous(), qkv[:, qd + kd:].contiguous(),
                                        a0_["k"], a0_["v"], pos, N_HEADS, N_KV, HEAD_DIM, FA, 0, m.cos, m.sin, 0)
    moe = (m.blocks[0].forward(h) if m.blocks[0] is not None else m.stack.layers[0].forward(h, FA, FW))[0]
    torch.cuda.synchronize()
    assert device.read_flags() == 0
    hn = h[:1].cpu().numpy()
    w = device.export_weight(a0_["wqkv"], qd + 2 * kd, nb, o.Q4_K)
    assert np.array_equal(qkv[:1].cpu().numpy(), onat.qk_linear(w, hn, qd + 2 * kd, nb, FW, o.Q4_K)), "EP decode: fused QKV"
    ck = a0_["k"][0, :, :pos + 1].cpu().numpy().astype(np.int64); cv = a0_["v"][0, :, :pos + 1].cpu().numpy().astype(np.int64)
    want = o.attention_cached(qkv[:1, :qd].cpu().numpy().reshape(1, N_HEADS, HEAD_DIM), ck, cv, pos, N_HEADS, N_KV, FA, None)
    assert np.array_equal(att[:1].cpu().numpy(), want), "EP decode: batched attention of sequence 0"
    if rank == 0:                                              # the other shards' weights exist on rank 0 only as a 1-block full stack
        from integer_inference_engine_b200.synth import SyntheticMoEStack
        full = SyntheticMoEStack(1, D_MODEL, E_FFN, N_EXPERTS, TOP_K, seed=1, fa=FA)
        _, ref = _oracle_rows(full, 0, hn)
        assert np.array_equal(moe[:1].cpu().numpy(), ref), "EP decode: MoE rows of block 0 differ from the oracle"
        for lay in full.layers:
            lay.close()
    m.tokens.copy_(torch.arange(rank * m.B, (rank + 1) * m.B, dtype=torch.int32, device="cuda") * 13 + 5)
    l0 = device.launch_count()
    m.capture()
    launches = (device.launch_count() - l0) // 2
    ms, clocks = _timed(lambda i: m.replay(), steps, warmup, world, local)
    assert device.read_flags() == 0
    ms_step = ms / steps
    peak, kind = measured_peak_gbs()
    # bytes one rank streams per step: its expert shard (every expert is touched at 64 x 8 routed pairs), the replicated
    # attention matrices and router, its sequences' visible cache rows, the head
    expert_b = (2 * E_FFN * nb * 144 + D_MODEL * (E_FFN // 256) * 210) * (N_EXPERTS // world)
    attn_b = (2 * qd + 2 * kd) * nb * 144 + N_EXPERTS * nb * 144
    kv_b = m.B * 2 * N_KV * (pos + 1) * HEAD_DIM * 4
    bytes_rank = args.layers * (expert_b + attn_b + kv_b) + VOCAB * nb * 210
    out = {"sequences": S, "ms_per_step": ms_step, "tok_per_s": S * 1e3 / ms_step, "parallelism": f"ep{world} x dp{world}",
           "layers": args.layers, "context": args.context, "step": "whole decode step (attention over per-sequence caches, "
           "expert-parallel MoE, head, picks) as one replayed CUDA graph at a fixed position",
           "exchange": ("all-gather dispatch + reduce-scatter combine per block (NCCL)" if world > 1 else "none (one rank)"),
           "a2a_bytes_per_rank_per_block": m.a2a_bytes_per_block, "gpu_launches_per_step": int(launches),
           "bytes_per_rank_per_step": bytes_rank, "hbm_frac_of_%s_peak" % kind: bytes_rank / (ms_step * 1e-3) / 1e9 / peak,
           "oracle_checked": "block 0: fused QKV, batched attention (sequence 0 of every rank), MoE rows (rank 0)", "clocks": clocks}
    del m
    return out


def run_ep_decode(args):
    rank, world, local = _dist_setup()
    res = ep_decode_measure(args, rank, world, local, args.steps, args.warmup)
    if rank == 0:
        cpu = None
        if args.cpu_sample_layers > 0:
            use_all_host_threads()
            step = CpuDecodeStep("port", 1, args.context)
            step.step(1)
            t0 = time.perf_counter(); step.step(1); t1 = time.perf_counter() - t0
            t0 = time.perf_counter(); step.step(0); th = time.perf_counter() - t0
            cpu = {"value": 1.0 / ((t1 - th) * args.layers + th), "unit": "tok/s", "cores": host_cores(), "kind": "port",
                   "sample": f"1 block and the head for ONE sequence, scaled to {args.layers} blocks (sequences are independent on the CPU)"}
        peak, kind = measured_peak_gbs()
        print(json.dumps({
            "metric": "decode_tok_per_s", "value": res["tok_per_s"], "unit": "tok/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": res["ms_per_step"], "higher_is_better": True, "scaling": "strong", "vs_baseline": None,
            "dtype": "int64", "data": "synthetic",
            "config": dict({"workload": f"config4_ep_decode: {res['sequences']} sequences x context {args.context}, {args.layers} blocks, "
                                        f"experts {N_EXPERTS // world}/rank, sequences {res['sequences'] // world}/rank",
                            "l2": "inputs larger than L2 (expert shard, caches and head streamed every step)"}, **res),
            "clocks": res["clocks"], "gpu_launches": res["gpu_launches_per_step"] * args.steps,
            "roofline": {"bound": "hbm", "kernel": "all kernels of one step on one rank (aggregate)", "unit": "GB/s", "peak": peak,
                         "peak_kind": kind, "achieved": res["bytes_per_rank_per_step"] / (res["ms_per_step"] * 1e-3) / 1e9,
                         "frac": res["bytes_per_rank_per_step"] / (res["ms_per_step"] * 1e-3) / 1e9 / peak, "traffic": None},
            "cpu_baseline": cpu}))
    import torch.distributed as dist
    if world > 1:
        dist.destroy_process_group()


def run_q1(args):
    """Q1_0 dense configuration (8B shape: 36 layers, d=4096, ffn 12288, vocab 151936): the seven linear
    products of every layer plus the output head, as a 512-token prefill pass and as batch-1 decode steps."""
    import torch

    from integer_inference_engine_b200 import device, q1_gpu
    from oracle import native as onat
    from oracle import qk_oracle as o
    rank, world, local = _dist_setup()
    assert world == 1, "the Q1_0 line is a single-GPU measurement"
    L = 36 if args.layers == 48 else args.layers
    d, ffn, vocab, frac = 4096, 12288, 151936, 16
    shapes = [("qkv", d + 2 * 1024, d), ("o", d, d), ("gate", ffn, d), ("up", ffn, d), ("down", d, ffn)]
    rng = np.random.default_rng(2)

    def make(out_f, in_f):
        bits = rng.integers(0, 256, size=(out_f, in_f // 128, 16), dtype=np.uint8)
        sc = np.rint(np.abs(rng.standard_normal((out_f, in_f // 128)) * 0.02).astype(np.float16).astype(np.float64) * (1 << frac))
        return bits, sc.astype(np.int32)
    layers, wbytes = [], 0
    first = None
    for li in range(L):
        hs = {}
        for name, of, inf in shapes:
            bits, sc = make(of, inf)
            hs[name] = q1_gpu.q1_register_weight(bits, sc)
            wbytes += of * (inf // 128) * 20
            if li == 0 and name == "gate":
                first = (bits, sc)
        layers.append(hs)
    hb, hsc = make(vocab, d)
    head = q1_gpu.q1_register_weight(hb, hsc)
    wbytes += vocab * (d // 128) * 20
    # parity: layer 0's gate projection on 3 rows against the checker
    xt = o.to_fixed(rng.standard_normal((3, d)), frac)
    got = q1_gpu.apply_dev(layers[0]["gate"], torch.from_numpy(xt).cuda(), frac).cpu().numpy()
    assert np.array_equal(got, onat.q1_linear(xt, first[0], first[1].astype(np.int64), frac)), "Q1_0 product differs from the oracle"

    def pass_(x_d, x_f, with_head):
        for hs in layers:
            q1_gpu.apply_dev(hs["qkv"], x_d, frac)
            q1_gpu.apply_dev(hs["o"], x_d, frac)
            q1_gpu.apply_dev(hs["gate"], x_d, frac)
            q1_gpu.apply_dev(hs["up"], x_d, frac)
            q1_gpu.apply_dev(hs["down"], x_f, frac)
        if with_head:
            q1_gpu.apply_dev(head, x_d[:1], frac)
    T = args.tokens or 512
    xd = torch.from_numpy(o.to_fixed(rng.standard_normal((T, d)), frac)).cuda()
    xf = torch.from_numpy(o.to_fixed(rng.standard_normal((T, ffn)), frac)).cuda()
    pf_ms, _ = _timed(lambda i: pass_(xd, xf, False), max(1, args.steps // 8), 1, 1, local)
    pf_ms /= max(1, args.steps // 8)
    x1, f1 = xd[:1].clone(), xf[:1].clone()
    pass_(x1, f1, True)                                           # sizes the scratch before capture
    torch.cuda.synchronize()
    l0 = device.launch_count()
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        with torch.cuda.graph(graph, stream=side):
            pass_(x1, f1, True)
    launches = device.launch_count() - l0
    ms, clocks = _timed(lambda i: graph.replay(), args.steps, args.warmup, 1, local)
    ms_step = ms / args.steps
    peak, kind = measured_peak_gbs()
    print(json.dumps({
        "metric": "decode_tok_per_s", "value": 1e3 / ms_step, "unit": "tok/s", "n_gpus": 1, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms_step, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "int64 modulo 2^64 via int8 digit planes", "data": "synthetic",
        "config": {"workload": f"config5_q1_linears: {L} layers x (qkv, o, gate, up, down) + head, batch-1 decode; "
                               f"attention, norms and the residual are not part of this line",
                   "prefill_tokens": T, "prefill_ms": pf_ms, "prefill_tok_per_s": T * 1e3 / pf_ms,
                   "l2": "inputs larger than L2: %d MB of weights per step" % (wbytes // 2**20)},
        "clocks": clocks, "gpu_launches": int(launches * args.steps),
        "roofline": {"bound": "hbm", "kernel": "q1 linears of one decode step (aggregate)", "achieved": wbytes / (ms_step * 1e-3) / 1e9,
                     "peak": peak, "peak_kind": kind, "unit": "GB/s", "frac": wbytes / (ms_step * 1e-3) / 1e9 / peak,
                     "traffic": None, "bytes_per_launch": wbytes}}))


def run_q1_token(args):
    """Whole decode token of the 1-bit decoder at the 8B shape (36 layers, d=4096, 32/8 heads of 128, ffn 12288,
    vocab 151936): Q1_0 embedding row, every layer's norms, fused QKV product, per-head norms, rotation, cached
    attention, O product, SwiGLU with wrapping products, down product, the Q1_0 head and the greedy pick, as one
    replayed CUDA graph; checked stage by stage on a small decoder against the CPU checker first."""
    import torch

    from integer_inference_engine_b200 import device
    from integer_inference_engine_b200.q1_model import SyntheticQ1Decoder
    from oracle import model_oracle
    rank, world, local = _dist_setup()
    assert world == 1, "the 1-bit decoder line is a single-GPU measurement"
    small = SyntheticQ1Decoder(n_layers=2, d_model=512, n_heads=8, n_kv=4, head_dim=64, d_ffn=768, vocab=640, context=20,
                               max_new=4, seed=3, keep_host=True)
    hl = [dict(L, k=L["k"].cpu().numpy().astype(np.int64), v=L["v"].cpu().numpy().astype(np.int64)) for L in small.host_layers]
    want, trace, logits = model_oracle.q1_decode_token(5, 20, hl, small.host_top, dict(d=512, H=8, Hkv=4, hd=64, ffn=768, frac=16),
                                                       small.cos.cpu().numpy(), small.sin.cpu().numpy())
    small.token.fill_(5)
    small.step(20)
    torch.cuda.synchronize()
    assert device.read_flags() == 0 and np.array_equal(small.x.cpu().numpy(), trace[-1:]) and int(small.token.item()) == want, \
        "1-bit decode token differs from the checker"
    del small
    L = 36 if args.layers == 48 else args.layers
    ctx = args.context if args.context else 512
    m = SyntheticQ1Decoder(n_layers=L, context=ctx, max_new=args.steps + args.warmup + 8, seed=2)
    m.token.fill_(11)
    l0 = device.launch_count()
    m.capture(ctx + args.steps + args.warmup + 4)
    launches = (device.launch_count() - l0) // 2
    ms, clocks = _timed(lambda i: m.replay(), args.steps, args.warmup, 1, local)
    ms_step = ms / args.steps
    assert device.read_flags() == 0
    tin = torch.zeros(1, dtype=torch.int32).pin_memory(); tout = torch.zeros(1, dtype=torch.int32).pin_memory()
    tin[0] = 11
    m.set_position(ctx)
    e2e_ms, _ = _timed(lambda i: m.decode_token(tin, tout), args.steps, 1, 1, local)
    wbytes = m.weight_bytes_per_token()
    kv = 2 * m.Hkv * m.hd * 4 * (ctx + args.warmup + args.steps // 2) * L
    peak, kind = measured_peak_gbs()
    print(json.dumps({
        "metric": "decode_tok_per_s", "value": 1e3 / ms_step, "unit": "tok/s", "n_gpus": 1, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms_step, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "int64 modulo 2^64 via int8 digit planes", "data": "synthetic",
        "config": {"workload": f"config5_q1_decode_token: {L} layers of the 8B 1-bit shape, whole token (embedding row, norms, QKV, "
                               f"per-head norms, RoPE, cached attention, O, SwiGLU, down, head, greedy pick), context {ctx}",
                   "l2": "inputs larger than L2: %d MB of weights per step" % (wbytes // 2**20)},
        "clocks": clocks, "gpu_launches": int(launches * args.steps),
        "e2e": {"value": 1e3 / (e2e_ms / args.steps), "unit": "tok/s", "h2d_bytes_per_step": 4, "d2h_bytes_per_step": 4},
        "roofline": {"bound": "hbm", "kernel": "all kernels of one decode token (aggregate)",
                     "achieved": (wbytes + kv) / (ms_step * 1e-3) / 1e9, "peak": peak, "peak_kind": kind, "unit": "GB/s",
                     "frac": (wbytes + kv) / (ms_step * 1e-3) / 1e9 / peak, "traffic": None, "bytes_per_launch": wbytes + kv}}))


_Q1_BRIDGE_PROBE = r'''
import json, sys, time
import numpy as np
from trinote.infer_int import gpu_native as g          # the reference's own bridge (baseline/_ref), library from BONSAI_BIN_DIR
assert g.gpu_available() and g.monolith_available(), "bridge reports the library unusable"
L, T, reps = int(sys.argv[1]), int(sys.argv[2]), int(sys.argv[3])
d, H, Hkv, hd, ffn, vocab, frac = 4096, 32, 8, 128, 12288, int(sys.argv[4]), 16
rng = np.random.default_rng(2)
def make(out_f, in_f):
    bits = rng.integers(0, 256, size=(out_f, in_f // 128, 16), dtype=np.uint8)
    sc = np.rint(np.abs(rng.standard_normal((out_f, in_f // 128)) * 0.02).astype(np.float16).astype(np.float64) * (1 << frac))
    return g.q1_register_weight(bits, sc.astype(np.int64))
gain = lambda n: g.buf_upload_i64(np.rint((np.abs(rng.standard_normal(n)) + 0.5) * (1 << frac)).astype(np.int64))
shapes = {"wq": (H * hd, d), "wk": (Hkv * hd, d), "wv": (Hkv * hd, d), "wo": (d, H * hd), "w1": (ffn, d), "wu": (ffn, d), "w2": (d, ffn)}
w = {k: [] for k in shapes}; gg = {k: [] for k in ("n1g", "n2g", "qng", "kng")}
for li in range(L):
    for k, (of, inf) in shapes.items():
        w[k].append(make(of, inf))
    gg["n1g"].append(gain(d)); gg["n2g"].append(gain(d)); gg["qng"].append(gain(hd)); gg["kng"].append(gain(hd))
w["out_head"], w["out_head_vocab"] = make(vocab, d), vocab
inv = 1.0 / (1e6 ** (np.arange(0, hd, 2) / hd)); ang = np.arange(T)[:, None] * inv[None, :]
gg["finalg"], gg["cos_h"], gg["sin_h"] = gain(d), g.buf_upload_i64(np.rint(np.cos(ang) * (1 << frac)).astype(np.int64)), \
    g.buf_upload_i64(np.rint(np.sin(ang) * (1 << frac)).astype(np.int64))
x = np.rint(rng.standard_normal((T, d)) * 0.05 * (1 << frac)).astype(np.int64)
inv_sqrt = round((1.0 / np.sqrt(hd)) * (1 << frac))
run = lambda: g.prefill_forward_gpu(x, (T, d, L, H, Hkv, hd, ffn), w, gg, frac, 1, inv_sqrt)
first = run()
assert first is not None, "the prefill reported overflow"
ts = []
for _ in range(reps):
    t0 = time.perf_counter(); run(); ts.append(time.perf_counter() - t0)
import hashlib
print(json.dumps({"ms_per_call": float(np.median(ts)) * 1e3, "calls": reps, "layers": L, "tokens": T,
                  "logits_sha256": hashlib.sha256(first.tobytes()).hexdigest(), "library": str(g._load_lib()._name)}))
'''


def q1_bridge_timing(lib_file: Path, layers: int, tokens: int, reps: int, vocab: int):
    """`bonsai_prefill_forward_gpu` called through the REFERENCE's own bridge module on a seeded model of the 8B layer
    shape, with `lib_file` as the `libbonsai_q1_gpu.so` it loads.  A child process per library."""
    import tempfile
    ref = ROOT / "baseline" / "_ref" / "bonsai"
    if not (ref / "src" / "trinote").exists() or not lib_file.exists():
        return {"unavailable": "reference 1-bit bridge or library not installed under baseline/_ref"}
    with tempfile.TemporaryDirectory() as tmp:
        os.symlink(lib_file, Path(tmp) / "libbonsai_q1_gpu.so")
        env = dict(os.environ)
        env["BONSAI_BIN_DIR"] = tmp
        env["BONSAI_NOTARY_HOME"] = tmp
        env["PYTHONPATH"] = str(ref / "src")
        try:
            run = subprocess.run([sys.executable, "-c", _Q1_BRIDGE_PROBE, str(layers), str(tokens), str(reps), str(vocab)],
                                 env=env, capture_output=True, text=True, timeout=900)
        except subprocess.TimeoutExpired:
            return {"unavailable": "timed out"}
    if run.returncode != 0:
        return {"unavailable": (run.stderr.strip().splitlines() or ["failed"])[-1][:200]}
    return json.loads(run.stdout.strip().splitlines()[-1])


def run_q1_prefill(args):
    """The 1-bit decoder's prefill through the reference's entry name `bonsai_prefill_forward_gpu` with HOST buffers (what
    `BonsaiReferenceModel.prefill_logits_gpu_resident` calls): 512 tokens through the layers of the 8B shape, last-row
    logits out.  Time is wall clock around the call (the entry synchronises; uploads and downloads are inside it).
    The same call is made through the reference's own bridge, once over the reference's CUDA library compiled for
    sm_100a and once over this one, on a bounded number of layers; the logits of the two must be the same bytes."""
    import torch

    from integer_inference_engine_b200 import device, q1_gpu
    from oracle import model_oracle
    rank, world, local = _dist_setup()
    assert world == 1, "the 1-bit prefill line is a single-GPU measurement"
    L = 36 if args.layers == 48 else args.layers
    T = args.tokens or 512
    d, H, Hkv, hd, ffn, vocab, frac = 4096, 32, 8, 128, 12288, 151936, 16
    rng = np.random.default_rng(2)

    def make(out_f, in_f):
        bits = rng.integers(0, 256, size=(out_f, in_f // 128, 16), dtype=np.uint8)
        sc = np.rint(np.abs(rng.standard_normal((out_f, in_f // 128)) * 0.02).astype(np.float16).astype(np.float64) * (1 << frac))
        return q1_gpu.q1_register_weight(bits, sc.astype(np.int32))
    gain = lambda n: q1_gpu.buf_upload_i64(np.rint((np.abs(rng.standard_normal(n)) + 0.5) * (1 << frac)).astype(np.int64))
    shapes = {"wq": (H * hd, d), "wk": (Hkv * hd, d), "wv": (Hkv * hd, d), "wo": (d, H * hd), "w1": (ffn, d), "wu": (ffn, d), "w2": (d, ffn)}
    w = {k: [] for k in shapes}
    g = {k: [] for k in ("n1g", "n2g", "qng", "kng")}
    wbytes = 0
    for li in range(L):
        for k, (of, inf) in shapes.items():
            w[k].append(make(of, inf))
            wbytes += of * (inf // 128) * 20
        g["n1g"].append(gain(d)); g["n2g"].append(gain(d)); g["qng"].append(gain(hd)); g["kng"].append(gain(hd))
    w["out_head"], w["out_head_vocab"] = make(vocab, d), vocab
    from integer_inference_engine_b200.model import rope_tables
    cos, sin = rope_tables(T, hd, 1e6, frac)
    g["finalg"], g["cos_h"], g["sin_h"] = gain(d), q1_gpu.buf_upload_i64(cos), q1_gpu.buf_upload_i64(sin)
    x = np.rint(rng.standard_normal((T, d)) * 0.05 * (1 << frac)).astype(np.int64)
    inv_sqrt = round((1.0 / np.sqrt(hd)) * (1 << frac))
    dims = (T, d, L, H, Hkv, hd, ffn)
    call = lambda: q1_gpu.prefill_forward_gpu(x, dims, w, g, frac, 1, inv_sqrt)
    l0 = device.launch_count()
    first = call()
    launches = device.launch_count() - l0
    assert first is not None, "the prefill reported overflow"
    for _ in range(args.warmup):
        call()
    ts = []
    with ClockSampler(local) as clk:
        for _ in range(args.steps):
            t0 = time.perf_counter(); out = call(); ts.append(time.perf_counter() - t0)
    clocks = clk.summary()
    assert np.array_equal(out, first)
    # wall-clock calls on a shared host: single calls are sometimes delayed several-fold by the host, so the line reports
    # the median call (the mean is kept beside it)
    ms, ms_mean = float(np.median(ts)) * 1e3, float(np.mean(ts)) * 1e3
    q1_gpu.q1_free_weights()
    torch.cuda.empty_cache()
    # kernel for kernel, through the reference's own bridge, on a bounded model (4 layers, small head)
    cmpL, cmpV = min(L, 4), 4096
    ref_lib = ROOT / "baseline" / "_ref" / "bin" / "reference_libbonsai_q1_gpu.so"
    theirs = q1_bridge_timing(ref_lib, cmpL, T, 3, cmpV)
    ours = q1_bridge_timing(ROOT / "integer_inference_engine_b200" / "lib" / "libbonsai_q1_gpu.so", cmpL, T, 3, cmpV)
    same = ("logits_sha256" in theirs and theirs.get("logits_sha256") == ours.get("logits_sha256"))
    peak, kind = measured_peak_gbs()
    macs = T * (wbytes // 20) * 128                          # one multiply-add per weight per token
    print(json.dumps({
        "metric": "prefill_tok_per_s", "value": T * 1e3 / ms, "unit": "tok/s", "n_gpus": 1, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": ms, "ms_per_step_mean": ms_mean, "timing": "median of the wall-clock calls", "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "int64 modulo 2^64 via int8 digit planes", "data": "synthetic",
        "config": {"workload": f"config5_q1_prefill: {T} tokens through {L} layers of the 8B 1-bit shape (norms, Q/K/V, per-head norms, "
                               f"RoPE, causal attention, O, SwiGLU, down) and the head on the last row, through "
                               f"bonsai_prefill_forward_gpu with host buffers",
                   "l2": "inputs larger than L2: %d MB of weights per pass" % (wbytes // 2**20),
                   "same_call_through_the_reference_bridge": {"layers": cmpL, "vocab": cmpV, "reference_cuda_library": theirs,
                                                              "this_library": ours, "logits_identical": bool(same)}},
        "clocks": clocks, "gpu_launches": int(launches * args.steps),
        "e2e": {"value": T * 1e3 / ms, "unit": "tok/s", "h2d_bytes_per_step": int(x.nbytes), "d2h_bytes_per_step": vocab * 8},
        "roofline": {"bound": "tensor", "kernel": "all kernels of one prefill pass (aggregate)", "unit": "TFLOP/s",
                     "achieved": 2 * macs * 8 / (ms * 1e-3) / 1e12, "peak": None, "frac": None, "traffic": None,
                     "note": "int8 digit-plane operations (8 planes per activation); the int8 peak is measured by the default workload"}}))


if __name__ == "__main__":
    a = parse()
    if a.impl == "reference":
        run_reference(a)
    elif a.workload == "prefill":
        run_prefill(a)
    elif a.workload == "ep_decode":
        run_ep_decode(a)
    elif a.workload == "q1":
        run_q1(a)
    elif a.workload == "q1_token":
        run_q1_token(a)
    elif a.workload == "q1_prefill":
        run_q1_prefill(a)
    else:
        run_ours(a)
