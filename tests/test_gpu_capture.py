"""Runs and stream capture: a captured run's replay gives the run's results (GPU)."""
import ctypes as C

import numpy as np
import pytest

import s615
import workloads as W

pytestmark = pytest.mark.gpu
FIELDS = ("calls", "gated", "probes", "pos", "hits", "tri_total", "tri_skipped")
torch = pytest.importorskip("torch")


def prepare(eng, arr, n):
    b = C.c_void_p()
    s615._check(s615.lib().s615_prepare(eng._ctx, C.cast(arr, C.c_void_p), n, C.byref(b)), "prepare")
    return b


def launch(eng, tid, b, stream):
    before = eng.launches
    s615._check(s615.lib().s615_run_batch(eng._ctx, tid, b, 0, C.c_void_p(stream.cuda_stream)), "run")
    return eng.launches - before


def results(eng, b):
    hits, nh, c = (s615.Hit * 65536)(), C.c_size_t(), s615.Counters()
    s615._check(s615.lib().s615_batch_results(eng._ctx, b, C.cast(hits, C.c_void_p), 65536,
                                              C.byref(nh), C.byref(c)), "results")
    h = s615.hits_to_array(hits, nh.value)
    a = np.stack([h[k].astype(np.uint64) for k in ("unit", "d", "e", "c4", "fp")], axis=1)
    return [getattr(c, f) for f in FIELDS], a[np.lexsort(a.T[::-1])].tolist()


def test_freeing_a_captured_batch(engine):
    """Replays give the run's results, and the calls after the batch is freed succeed."""
    N = 715
    tid = engine.build_table(N, 16)
    try:
        arr, n = W.unit_array(W.cls5_units(1000, 30000), W.plants(4, 0, 1000, 30000, N), N)
        p, st = prepare(engine, arr, n), torch.cuda.Stream()
        launch(engine, tid, p, st)
        torch.cuda.synchronize()
        want = results(engine, p)
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            launch(engine, tid, p, st)
        for _ in range(2):
            g.replay()
        torch.cuda.synchronize()
        assert results(engine, p) == want and want[0][2] > 0
        del g
        assert s615.lib().s615_batch_free(engine._ctx, p) == 0
        engine.free_table(engine.build_table(300, 16))
        h, c = engine.run(tid, arr, n)
        assert [getattr(c, f) for f in FIELDS] == want[0] and len(h) == len(want[1])
    finally:
        engine.free_table(tid)


@pytest.fixture(scope="module")
def staged():
    """A table whose large batches are probed in stages, and such a batch's units."""
    N = 40000
    arr, n = W.unit_array(W.cls5_units(1650000, 1650600)[:1500], W.plants(2, 5, 1600000, 1680000, N), N)
    with s615.Engine(0) as eng:
        yield eng, eng.build_table(N, 20), arr, n


def give_space_back(eng):
    eng.free_table(eng.build_table(300, 16))


def test_beside_a_capture(staged):
    """The first staged run of a context while another stream is captured in the default
    (global) mode: the capture stays valid, and the run is staged."""
    eng, tid, arr, n = staged
    p, st = prepare(eng, arr, n), torch.cuda.Stream()
    launch(eng, tid, p, st)                   # kernels loaded
    torch.cuda.synchronize()
    want = results(eng, p)
    give_space_back(eng)
    x, g = torch.ones(1000, device="cuda"), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        y = x + 1
        launched = launch(eng, tid, p, st)
    g.replay()
    torch.cuda.synchronize()
    assert launched >= 5 and float(y.sum()) == 2000
    assert results(eng, p) == want
    s615.lib().s615_batch_free(eng._ctx, p)


def test_a_captured_run_is_direct(staged):
    """A run on a stream that is being captured goes without the space, and its replay
    gives the staged run's results."""
    eng, tid, arr, n = staged
    p, st = prepare(eng, arr, n), torch.cuda.Stream()
    assert launch(eng, tid, p, st) >= 5
    torch.cuda.synchronize()
    want, g = results(eng, p), torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        assert launch(eng, tid, p, st) <= 2
    give_space_back(eng)
    for _ in range(2):
        g.replay()
    torch.cuda.synchronize()
    assert results(eng, p) == want
    del g
    s615.lib().s615_batch_free(eng._ctx, p)
