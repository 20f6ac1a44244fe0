"""Host work shared among threads where the system does not give all of them: the work is done, nothing is thrown out of the call and
no thread is left behind.  Needs g++, no GPU."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    so = tmp_path_factory.mktemp("host_threads") / "libhost_threads.so"
    build = subprocess.run([gxx, "-O2", "-std=c++17", "-shared", "-fPIC", "-pthread", "-I", str(ROOT / "integer_inference_engine_b200" / "csrc"),
                            str(ROOT / "tests" / "host_threads_check.cpp"), "-o", str(so)], capture_output=True, text=True, timeout=600)
    assert build.returncode == 0, build.stderr[-2000:]
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("made", [0, 1, 2, 3])
def test_every_piece_once_with_the_threads_there_are(lib, made):
    marks = np.zeros(10_000, np.int32)
    assert lib.h_share(made, marks.size, marks.ctypes.data_as(ctypes.POINTER(ctypes.c_int))) == made + 1
    assert (marks == 1).all()
