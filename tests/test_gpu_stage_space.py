"""The staged probe's space: taken once and not grown by waiting and freeing, also while
serving (GPU)."""
import ctypes as C
import time

import numpy as np
import pytest

import s615
import workloads as W
from test_gpu_staged import FIELDS, rows

pytestmark = pytest.mark.gpu
N = 40000
MB = 1 << 20
torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def table():
    with s615.Engine(0) as eng:
        yield eng, eng.build_table(N, 20)


@pytest.fixture()
def no_space(table):
    """The table, with whatever an earlier run kept given back."""
    eng, tid = table
    eng.free_table(eng.build_table(300, 16))
    return eng, tid


def units(B, n):
    return W.unit_array(W.cls5_units(B, B + n)[:n], W.plants(2, B, 1600000, 1680000, N), N)


def mem_free(eng):
    f, t = C.c_size_t(), C.c_size_t()
    s615._check(s615.lib().s615_mem_info(eng._ctx, C.byref(f), C.byref(t)), "mem_info")
    return f.value


def prepare(eng, arr, n):
    b = C.c_void_p()
    s615._check(s615.lib().s615_prepare(eng._ctx, C.cast(arr, C.c_void_p), n, C.byref(b)), "prepare")
    return b


def launch(eng, tid, b, stream):
    before = eng.launches
    s615._check(s615.lib().s615_run_batch(eng._ctx, tid, b, 0, C.c_void_p(stream.cuda_stream)), "run")
    return eng.launches - before


def sorted_rows(h):
    a = rows(h)
    return a[np.lexsort(a.T[::-1])].tolist()


def results(eng, b):
    hits, nh, c = (s615.Hit * 65536)(), C.c_size_t(), s615.Counters()
    s615._check(s615.lib().s615_batch_results(eng._ctx, b, C.cast(hits, C.c_void_p), 65536,
                                              C.byref(nh), C.byref(c)), "results")
    return [getattr(c, f) for f in FIELDS], sorted_rows(s615.hits_to_array(hits, nh.value))


def direct(eng, tid, arr, n, piece=100):
    """Counters and hits of the units in pieces that are probed directly."""
    ctr, hits = np.zeros(len(FIELDS), dtype=np.int64), []
    for lo in range(0, n, piece):
        part = (s615.Unit * min(piece, n - lo))(*[arr[i] for i in range(lo, min(n, lo + piece))])
        before = eng.launches
        h, c = eng.run(tid, part, len(part))
        assert eng.launches - before <= 4
        hits.append(rows(h, lo))
        ctr += [getattr(c, f) for f in FIELDS]
    hits = np.concatenate(hits)
    return ctr.tolist(), hits[np.lexsort(hits.T[::-1])].tolist()


def test_a_larger_run_does_not_wait(no_space):
    """A run that wants more space than the one before launches while that one's work is
    still on the device."""
    eng, tid = no_space
    a, b = units(1670000, 1300), units(1640000, 4000)
    pa, pb = prepare(eng, *a), prepare(eng, *b)
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    assert launch(eng, tid, pa, s1) >= 5
    held = mem_free(eng)
    for _ in range(30):
        launch(eng, tid, pa, s1)
    ev = torch.cuda.Event()
    ev.record(s1)
    assert launch(eng, tid, pb, s2) >= 5
    assert not ev.query()              # a hundred milliseconds of work before it
    assert mem_free(eng) >= held - 2 * MB
    torch.cuda.synchronize()
    got = results(eng, pb)
    for p in (pa, pb):
        s615.lib().s615_batch_free(eng._ctx, p)
    assert got == direct(eng, tid, *b)


def test_serving_reaches_the_stages(no_space):
    """Requests large enough for the stages, each larger than the one before: their hits
    are those of the direct probe, and the space is taken once."""
    eng, tid = no_space
    reqs = [units(1670000, 600), units(1660000, 1300), units(1640000, 4000)]
    want = [direct(eng, tid, *r)[1] for r in reqs]
    eng.free_table(eng.build_table(300, 16))
    eng.serve_start(2)
    try:
        free, done = [], []
        for arr, n in reqs:
            before = eng.launches
            t = eng.submit(tid, arr, n)
            got, end = [], time.time() + 60
            while not got and time.time() < end:
                got = eng.poll(4, 1000)
            assert got and got[0]["ticket"] == t and got[0]["status"] == 0
            assert eng.launches - before >= 5
            done.append(sorted_rows(got[0]["hits"]))
            free.append(mem_free(eng))
    finally:
        eng.serve_stop()
    assert done == want
    assert free[0] - free[2] < 100 * MB   # unit records and items alone


def test_less_room_then_more(table):
    """A space that little room made small is given up for a larger one when the budget and
    an idle device let it."""
    eng, tid = table
    arr, n = units(1640000, 4000)
    lib = s615.lib()
    cells = eng.table_info(tid).device_bytes
    seen = []
    for budget in (cells + (7 << 30), 0):
        s615._check(lib.s615_set_budget(eng._ctx, budget), "set_budget")
        if not seen:
            eng.free_table(eng.build_table(300, 16))   # whatever an earlier run kept
        before = eng.launches
        h, c = eng.run(tid, arr, n)
        seen.append((eng.launches - before, [getattr(c, f) for f in FIELDS], sorted_rows(h)))
    assert seen[0][1:] == seen[1][1:]
    assert seen[0][0] > seen[1][0] >= 5       # more chunks of less space
