"""The gated product of an expert, ((g * sigmoid(g)) >> fa) * u >> fa, as the tiles' epilogue evaluates it (32-bit form up to a
scale of 2^24, general form beyond), compiled for the CPU and compared with the NumPy checker.  Needs nvcc, no GPU."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from oracle import native as onat
from oracle import qk_oracle as o

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not found")
    so = tmp_path_factory.mktemp("host_silu") / "libhost_silu.so"
    build = subprocess.run([nvcc, "-O2", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-shared", "-Xcompiler", "-fPIC",
                            "-I", str(ROOT / "integer_inference_engine_b200" / "csrc"), str(ROOT / "tests" / "host_silu_check.cu"),
                            "-o", str(so)], capture_output=True, text=True, timeout=600)
    assert build.returncode == 0, build.stderr[-2000:]
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("fa", [8, 16, 17, 24, 25])
def test_gated_product(lib, fa):
    rng = np.random.default_rng(fa)
    clip = ((fa + 2) << (2 * fa)) // int(o._scaled_log2e(fa))
    edges = np.array([0, 1, -1, clip - 1, clip, clip + 1, -clip, -clip - 1, 1 << fa, -(1 << fa), 1 << 40, -(1 << 40)], np.int64)
    g = np.concatenate([edges] + [rng.integers(-(1 << b), 1 << b, size=20_000, dtype=np.int64) for b in (fa, fa + 4, 2 * fa, 33, 48)])
    u = rng.integers(-(1 << 40), 1 << 40, size=g.size, dtype=np.int64)
    y = np.empty_like(g)
    p = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_int64))
    lib.h_silu_up(p(g), p(u), p(y), ctypes.c_longlong(g.size), fa)
    small = np.abs(g) < (1 << 46)
    want = [(int(s) * int(v)) >> fa for s, v in zip(o.silu_int(g[small], fa), u[small])]
    assert [int(v) for v in y[small]] == [((w + (1 << 63)) % (1 << 64)) - (1 << 63) for w in want]


@pytest.mark.parametrize("fa", [1, 8, 14, 15, 16, 24, 25])
def test_gated_product_of_the_least_int64(lib, fa):
    """The distance of INT64_MIN from zero wraps in the sigmoid, as NumPy's does."""
    g = np.array([np.iinfo(np.int64).min, np.iinfo(np.int64).min + 1, np.iinfo(np.int64).max], np.int64)
    u, y = np.full(3, 3, np.int64), np.empty(3, np.int64)
    p = lambda a: a.ctypes.data_as(ctypes.POINTER(ctypes.c_int64))
    lib.h_silu_up_any(p(g), p(u), p(y), ctypes.c_longlong(3), fa)
    sig = onat.sigmoid(g, fa)
    wrapped = lambda v: (v + (1 << 63)) % (1 << 64) - (1 << 63)
    assert list(y) == [wrapped((((int(a) * int(b)) >> fa) * 3) >> fa) for a, b in zip(g, sig)]
