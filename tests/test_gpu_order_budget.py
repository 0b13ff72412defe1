"""Items that would be ordered on the device are ordered on the host where the budget has
no room for a second copy of them (GPU)."""
import ctypes as C

import numpy as np
import pytest

import s615

pytestmark = pytest.mark.gpu
FIELDS = ("calls", "gated", "probes", "pos", "hits", "tri_total", "tri_skipped")


def prepare(eng, arr, n):
    b, items = C.c_void_p(), C.c_size_t()
    s615._check(s615.lib().s615_prepare(eng._ctx, C.cast(arr, C.c_void_p), n, C.byref(b)), "prepare")
    s615.lib().s615_batch_size(b, None, C.byref(items), None)
    return b, items.value


def results(eng, tid, b):
    hits, nh, c = (s615.Hit * 65536)(), C.c_size_t(), s615.Counters()
    s615._check(s615.lib().s615_run_batch(eng._ctx, tid, b, 0, None), "run")
    s615._check(s615.lib().s615_batch_results(eng._ctx, b, C.cast(hits, C.c_void_p), 65536,
                                              C.byref(nh), C.byref(c)), "results")
    h = s615.hits_to_array(hits, nh.value)
    a = np.stack([h[k].astype(np.uint64) for k in ("unit", "d", "e", "c4", "fp")], axis=1)
    return [getattr(c, f) for f in FIELDS], a[np.lexsort(a.T[::-1])].tolist()


def test_no_room_for_a_second_copy():
    N = 4800
    arr, n = s615.candidates617(200003)
    n = min(n, 30)
    with s615.Engine(0) as eng:
        tid = eng.build_table(N, 16)
        b, items = prepare(eng, arr, n)
        assert items > 1 << 14
        want = results(eng, tid, b)
        assert want[0][2] > 0 and want[1]
        s615.lib().s615_batch_free(eng._ctx, b)
        eng.free_table(eng.build_table(300, 16))   # whatever is kept is given back
        # the table, the gate patterns, and the batch's own buffers: records, items,
        # counters, hits
        held = eng.table_info(tid).device_bytes + 4 * (4 * 660 + 400 + 2 * 7839)
        own = 224 * n + 8 * items + 112 + 32 * (1 << 20)
        s615._check(s615.lib().s615_set_budget(eng._ctx, held + own + (64 << 10)), "set_budget")
        b, again = prepare(eng, arr, n)
        assert again == items and 8 * items > 64 << 10
        assert results(eng, tid, b) == want
        s615.lib().s615_batch_free(eng._ctx, b)
