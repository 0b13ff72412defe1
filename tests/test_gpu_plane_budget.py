"""Planes and the HBM budget: a table's planes are taken only from room that is there,
and are given back before an allocation that needs the room fails (GPU)."""
import ctypes as C

import numpy as np
import pytest

import s615
import workloads as W

pytestmark = pytest.mark.gpu
N, R = 9000, 16      # 4-byte cells, an 8-bit plane of a quarter of their size
MB = 1 << 20
FIELDS = ("calls", "gated", "probes", "pos", "hits")


def set_budget(eng, b):
    s615._check(s615.lib().s615_set_budget(eng._ctx, b), "set_budget")


def key(h, c):
    a = np.stack([h[k].astype(np.uint64) for k in ("unit", "d", "e", "c4", "fp")], axis=1)
    return [getattr(c, f) for f in FIELDS], a[np.lexsort(a.T[::-1])].tolist()


@pytest.fixture(scope="module")
def saved(tmp_path_factory):
    """(path, cells) of a table file; units whose B it covers."""
    path = str(tmp_path_factory.mktemp("plane") / "t.bin")
    with s615.Engine(0) as eng:
        tid = eng.build_table(N, R)
        eng.save_table(tid, path)
        m = eng.table_info(tid).hdr.m_cells
        assert eng.table_info(tid).device_bytes == 4 * m + m // 4 * 4 + (4 if m % 4 else 0)
    arr, n = W.unit_array(W.cls5_units(200000, 200060), W.plants(5, 3, 190000, 200060, N), N)
    return path, m, arr, n


def test_run_takes_the_planes_room(saved):
    path, m, arr, n = saved
    with s615.Engine(0) as eng:
        tid = eng.load_table(path, N, s615.LAYOUT_WIDE)
        want = key(*eng.run(tid, arr, n))
        with s615.Engine(0) as other:   # nothing kept of an earlier run
            t2 = other.load_table(path, N, s615.LAYOUT_WIDE)
            # room for the run's buffers (32 MB of hits) beside the cells, not beside the plane
            set_budget(other, 4 * m + 60 * MB)
            assert other.table_info(t2).device_bytes > 4 * m
            for _ in range(2):
                assert key(*other.run(t2, arr, n)) == want
            assert other.table_info(t2).device_bytes == 4 * m


def test_second_table_takes_the_planes_room(saved):
    path, m, arr, n = saved
    packed = (m * R + 7) // 8
    with s615.Engine(0) as eng:
        t1 = eng.load_table(path, N, s615.LAYOUT_WIDE)
        want = key(*eng.run(t1, arr, n))
        set_budget(eng, 4 * m + packed + 42 * MB)
        t2 = eng.load_table(path, N, s615.LAYOUT_PACKED)
        assert eng.table_info(t1).device_bytes == 4 * m
        assert key(*eng.run(t1, arr, n)) == want
        assert key(*eng.run(t2, arr, n)) == want


def test_auto_layout_counts_the_planes_room(saved):
    path, m, arr, n = saved
    packed = (m * R + 7) // 8
    with s615.Engine(0) as eng:
        t1 = eng.load_table(path, N, s615.LAYOUT_WIDE)
        set_budget(eng, 8 * m + packed + (4 << 30) + 12 * MB)
        t2 = eng.load_table(path, N, s615.LAYOUT_AUTO)
        assert eng.table_info(t2).layout == s615.LAYOUT_WIDE
        assert eng.table_info(t1).device_bytes == 4 * m
        assert key(*eng.run(t1, arr, n)) == key(*eng.run(t2, arr, n))


def test_no_stage_plane_without_room_for_the_stages(tmp_path):
    """The 4-bit plane of the staged probe only where the budget has room for the stages'
    own space beside it; the first plane all the same."""
    N, path = 25001, str(tmp_path / "t.bin")
    with s615.Engine(0) as eng:
        tid = eng.build_table(N, R)
        info = eng.table_info(tid)
        m = info.hdr.m_cells
        plane = lambda bits: (m + 32 // bits - 1) // (32 // bits) * 4
        assert info.device_bytes == 4 * m + plane(1) + plane(2) + plane(4)
        eng.save_table(tid, path)
    cells = ((m * R + 7) // 8 + 8 + 7) // 8 * 8 + 8   # the file form of the cells, in whole words and one more
    with s615.Engine(0, cells + (1 << 30)) as eng:
        tid = eng.load_table(path, N, s615.LAYOUT_PACKED)
        assert eng.table_info(tid).device_bytes == cells + plane(2)


def test_planes_of_a_captured_run_stay(saved):
    """A run that is being captured leaves its table's plane in a graph: the plane is then
    not given back, and the graph's replay gives the run's results."""
    torch = pytest.importorskip("torch")
    path, m, arr, n = saved
    lib = s615.lib()
    with s615.Engine(0) as eng:
        tid = eng.load_table(path, N, s615.LAYOUT_WIDE)
        want = key(*eng.run(tid, arr, n))
        b = C.c_void_p()
        s615._check(lib.s615_prepare(eng._ctx, C.cast(arr, C.c_void_p), n, C.byref(b)), "prepare")
        st, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st):
            s615._check(lib.s615_run_batch(eng._ctx, tid, b, 0, C.c_void_p(st.cuda_stream)), "run")
        held = eng.table_info(tid).device_bytes
        assert held > 4 * m
        set_budget(eng, held + 8 * MB)
        with pytest.raises(s615.S615Error) as e:   # needs the plane's room and does not get it
            eng.load_table(path, N, s615.LAYOUT_PACKED)
        assert e.value.status == -6
        assert eng.table_info(tid).device_bytes == held
        g.replay()
        torch.cuda.synchronize()
        hits, nh, c = (s615.Hit * 65536)(), C.c_size_t(), s615.Counters()
        s615._check(lib.s615_batch_results(eng._ctx, b, C.cast(hits, C.c_void_p), 65536, C.byref(nh),
                                           C.byref(c)), "results")
        assert key(s615.hits_to_array(hits, nh.value), c) == want
        del g
        lib.s615_batch_free(eng._ctx, b)
