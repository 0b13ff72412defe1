"""No launch takes L2 from the rest of the process (GPU)."""
import ctypes as C

import pytest

import s615
import workloads as W

pytestmark = pytest.mark.gpu
LIMIT_PERSISTING_L2 = 0x06       # cudaLimitPersistingL2CacheSize


@pytest.mark.parametrize("N,r", [(715, 48), (1600, 48), (5000, 48)])
def test_a_peel_leaves_the_l2_set_aside_alone(engine, N, r):
    # tables of 2.5 and 13 MB and one past the set-aside the device offers (125 MB)
    pytest.importorskip("torch")
    rt = C.CDLL("libcudart.so.12")
    rt.cudaDeviceGetLimit.argtypes = [C.POINTER(C.c_size_t), C.c_int]
    before, after = C.c_size_t(1), C.c_size_t(2)
    assert rt.cudaDeviceGetLimit(C.byref(before), LIMIT_PERSISTING_L2) == 0
    tid = engine.build_table(N, r)
    try:
        arr, n = W.unit_array(W.cls5_units(42 * N - 200, 42 * N), [], N)
        h0, c0 = engine.cls5_run(tid, arr, n)
        h1, c1 = engine.cls5_run(tid, arr, n, flags=s615.F_NO_L2_WINDOW)
    finally:
        engine.free_table(tid)
    assert (c0.calls, c0.gated, c0.probes, c0.hits) == (c1.calls, c1.gated, c1.probes, c1.hits)
    assert rt.cudaDeviceGetLimit(C.byref(after), LIMIT_PERSISTING_L2) == 0
    assert after.value == before.value
