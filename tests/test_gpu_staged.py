"""The staged probe of large batches gives the direct probe's hits and counters:
the same units in one run past its threshold and in runs below it (GPU)."""
import ctypes as C

import numpy as np
import pytest

import s615
import workloads as W

pytestmark = pytest.mark.gpu
N = 40000            # the smallest tables past L2 are probed in stages
KEYS = 1e8           # from 2.5e7 keys; these batches hold more, their pieces fewer
FIELDS = ("calls", "gated", "probes", "pos", "hits", "tri_total", "tri_skipped")


@pytest.fixture(scope="module", params=[(20, s615.LAYOUT_WIDE), (18, s615.LAYOUT_PACKED)])
def staged_table(request):
    eng = s615.Engine(0)
    tid = eng.build_table(N, *request.param)
    yield eng, tid
    eng.close()


def rows(h, base=0):
    a = np.stack([h[k].astype(np.uint64) for k in ("unit", "d", "e", "c4", "fp")], axis=1)
    a[:, 0] += np.uint64(base)
    return a


def run_pieces(eng, tid, arr, n, piece, flags=0):
    ctr, hits = np.zeros(len(FIELDS), dtype=np.int64), []
    sz = C.sizeof(s615.Unit)
    for lo in range(0, n, piece):
        k = min(piece, n - lo)
        part = (s615.Unit * k)()
        C.memmove(part, C.byref(arr, lo * sz), k * sz)
        before = eng.launches
        h, c = eng.run(tid, part, k, flags)
        assert eng.launches - before <= 4        # packing, then one launch or two
        hits.append(rows(h, lo))
        ctr += [getattr(c, f) for f in FIELDS]
    return np.concatenate(hits), ctr


def check(eng, tid, arr, n, piece, flags=0):
    before = eng.launches
    h, c = eng.run(tid, arr, n, flags)
    assert eng.launches - before >= 5            # emit, three stages, resolve
    want_h, want_c = run_pieces(eng, tid, arr, n, piece, flags)
    got = rows(h)
    assert c.probes >= KEYS or flags
    np.testing.assert_array_equal([getattr(c, f) for f in FIELDS], want_c)
    np.testing.assert_array_equal(got[np.lexsort(got.T[::-1])], want_h[np.lexsort(want_h.T[::-1])])
    assert len(got) > 0
    return got


def test_class5(staged_table):
    eng, tid = staged_table
    units = W.cls5_units(1675000, 1675600)[:1701]
    plants = W.plants(9, 4, 1600000, 1680000, N)
    arr, n = W.unit_array(units, plants, N)
    got = check(eng, tid, arr, n, 100)
    for j, p in enumerate(plants):
        assert ((got[:, 0] == len(units) + j) & (got[:, 4] == np.uint64(p.fp))).any()


@pytest.mark.parametrize("N,bits,first,n", [(34000, 1, 0, 1501), (28000, 1, 1, 2000),
                                            (25001, 2, 1, 2600)])
def test_table_with_planes_of_its_own(N, bits, first, n):
    """A table with a plane of 1 or 2 bits: the keys go through one of one bit, if it is
    small enough (perhaps that plane), into the stages, which compare the next four."""
    with s615.Engine(0) as eng:
        tid = eng.build_table(N, 20)
        info = eng.table_info(tid)
        m = info.hdr.m_cells
        plane = lambda k: (m + 32 // k - 1) // (32 // k) * 4 if k else 0
        own = plane(first) if first != bits else 0
        assert info.device_bytes == 4 * m + plane(bits) + own + plane(4)
        B = 42 * N - 3000
        plants = W.plants(9, 4, B - 90000, B, N)
        arr, k = W.unit_array(W.cls5_units(B, B + 2900)[:n], plants, N)
        got = check(eng, tid, arr, k, 100)
        for j, p in enumerate(plants):
            assert ((got[:, 0] == k - len(plants) + j) & (got[:, 4] == np.uint64(p.fp))).any()


def test_no_gate(staged_table):
    eng, tid = staged_table
    arr, n = W.unit_array(W.cls5_units(1675000, 1675040)[:41], [], N)
    check(eng, tid, arr, n, 2, s615.F_NO_GATE)


def test_mixed_kinds_in_one_batch(staged_table):
    eng, tid = staged_table
    units = W.mixed_units(2200, 5, 1200000, 1680000)
    arr, n = W.mixed_unit_array(units, W.plants(3, 1, 1200000, 1680000, N),
                                W.plants234(4, 2, 1200000, 1680000, N), N)
    jobs, nj, _ = s615.expand_units([x for x in units if x[0] in (2, 4)][:40])
    cands, nc = s615.candidates617(54347)
    both = (s615.Unit * (n + nj + nc))()
    sz = C.sizeof(s615.Unit)
    C.memmove(both, arr, n * sz)
    C.memmove(C.byref(both, n * sz), jobs, nj * sz)
    C.memmove(C.byref(both, (n + nj) * sz), cands, nc * sz)
    check(eng, tid, both, n + nj + nc, 150)


def test_chunks_past_their_pages():
    """Little HBM left, so several chunks, and the heavy units first, so that the
    first chunk holds far more keys than its pages: the rest is probed directly."""
    heavy, light = W.cls5_units(1675000, 1675700)[:1901], W.cls5_units(60000, 72000)[:10000]
    arr, n = W.unit_array(heavy + light, [], N)
    with s615.Engine(0) as eng:
        tid = eng.build_table(N, 20)
        s615._check(s615.lib().s615_set_budget(
            eng._ctx, eng.table_info(tid).device_bytes + (9 << 30)), "set_budget")
        before = eng.launches
        eng.run(tid, arr, n)
        assert eng.launches - before > 5         # more than one chunk
        check(eng, tid, arr, n, 100)


def test_two_streams_share_the_space(staged_table):
    torch = pytest.importorskip("torch")
    eng, tid = staged_table
    lib = s615.lib()
    a = W.unit_array(W.cls5_units(1675000, 1675600)[:1500], [], N)
    b = W.unit_array(W.cls5_units(1640000, 1640600)[:1600], [], N)
    streams, batches = [torch.cuda.Stream() for _ in range(2)], []
    for arr, n in (a, b):
        p = C.c_void_p()
        s615._check(lib.s615_prepare(eng._ctx, C.cast(arr, C.c_void_p), n, C.byref(p)), "prepare")
        batches.append(p)
    for p, st in zip(batches, streams):
        s615._check(lib.s615_run_batch(eng._ctx, tid, p, 0, C.c_void_p(st.cuda_stream)), "run")
    torch.cuda.synchronize()
    for p, (arr, n) in zip(batches, (a, b)):
        hits, nh, c = (s615.Hit * 65536)(), C.c_size_t(), s615.Counters()
        s615._check(lib.s615_batch_results(eng._ctx, p, C.cast(hits, C.c_void_p), 65536, C.byref(nh),
                                           C.byref(c)), "results")
        got = rows(s615.hits_to_array(hits, nh.value))
        lib.s615_batch_free(eng._ctx, p)
        want_h, want_c = run_pieces(eng, tid, arr, n, 100)
        np.testing.assert_array_equal([getattr(c, f) for f in FIELDS], want_c)
        np.testing.assert_array_equal(got[np.lexsort(got.T[::-1])],
                                      want_h[np.lexsort(want_h.T[::-1])])
