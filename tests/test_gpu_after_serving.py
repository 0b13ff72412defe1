"""After the serving loop has stopped, batches are packed on the device again (GPU)."""
import ctypes as C

import pytest

import s615
import workloads as W

pytestmark = pytest.mark.gpu


def copied(eng, arr, n):
    """Host-to-device bytes of preparing n units: 72 a unit when the device packs them."""
    lib, b, nb = s615.lib(), C.c_void_p(), C.c_size_t()
    s615._check(lib.s615_prepare(eng._ctx, C.cast(arr, C.c_void_p), n, C.byref(b)), "prepare")
    lib.s615_batch_size(b, None, None, C.byref(nb))
    lib.s615_batch_free(eng._ctx, b)
    return nb.value


def test_device_packing_after_a_session():
    N = 715
    arr, n = W.unit_array(W.cls5_units(1000, 30000)[:200], [], N)
    with s615.Engine(0) as eng:
        tid = eng.build_table(N, 20)
        assert copied(eng, arr, n) == 72 * n
        eng.serve_start(2)
        ticket = eng.submit(tid, arr, n)
        got = []
        while not got:
            got = eng.poll(4, 1000)
        assert got[0]["ticket"] == ticket and got[0]["status"] == 0
        eng.serve_stop()
        assert copied(eng, arr, n) == 72 * n
