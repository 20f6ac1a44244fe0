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
