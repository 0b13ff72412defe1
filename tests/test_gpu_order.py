"""Work items put in order on the device: a batch with enough (6,1,7) items gives
the counters and hits of the same units in batches ordered on the host (GPU)."""
import ctypes as C

import numpy as np
import pytest

import s615

pytestmark = pytest.mark.gpu
FIELDS = ("calls", "gated", "probes", "pos", "hits", "tri_total", "tri_skipped")


def rows(h, base=0):
    a = np.stack([h[k].astype(np.uint64) for k in ("unit", "d", "e", "c4", "fp")], axis=1)
    a[:, 0] += np.uint64(base)
    return a


def run(eng, tid, arr, lo, n, flags=0):
    part = (s615.Unit * n)()
    C.memmove(part, C.byref(arr, lo * C.sizeof(s615.Unit)), n * C.sizeof(s615.Unit))
    b, items = C.c_void_p(), C.c_size_t()
    s615._check(s615.lib().s615_prepare(eng._ctx, C.cast(part, C.c_void_p), n, C.byref(b)), "prepare")
    s615.lib().s615_batch_size(b, None, C.byref(items), None)
    s615.lib().s615_batch_free(eng._ctx, b)
    h, c = eng.run(tid, part, n, flags)
    return rows(h, lo), np.array([getattr(c, f) for f in FIELDS], dtype=np.int64), items.value


@pytest.mark.parametrize("make", ["jobs", "candidates"])
def test_device_order(engine, make):
    if make == "jobs":
        N, piece = 970, 2500
        arr, n = s615.jobs617_band([B for B in range(40001, 40200) if B % 2 and B % 3 and B % 7],
                                   (2, 3, 4))
    else:
        N, piece = 4800, 8
        arr, n = s615.candidates617(200003)
        n = min(n, 30)
    tid = engine.build_table(N, 16)
    try:
        got, ctr, items = run(engine, tid, arr, 0, n)
        assert items > 1 << 14
        want, tot = [], np.zeros(len(FIELDS), dtype=np.int64)
        for lo in range(0, n, piece):
            h, c, few = run(engine, tid, arr, lo, min(piece, n - lo))
            assert few <= 1 << 14
            want.append(h)
            tot += c
        want = np.concatenate(want)
        np.testing.assert_array_equal(ctr, tot)
        assert len(got) > 0
        np.testing.assert_array_equal(got[np.lexsort(got.T[::-1])], want[np.lexsort(want.T[::-1])])
        if make == "candidates":   # the plain form goes unit by unit through the host's order
            h, c, _ = run(engine, tid, arr, 0, n, s615.F_PLAIN)
            np.testing.assert_array_equal(c, tot)
            np.testing.assert_array_equal(h[np.lexsort(h.T[::-1])], want[np.lexsort(want.T[::-1])])
    finally:
        engine.free_table(tid)
