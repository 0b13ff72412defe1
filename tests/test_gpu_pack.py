"""Unit records and work items made on the device give what the host's give: the
same units run alone (packed on the device) and with a class-7 unit beside them,
which sends the whole batch the host's way (GPU)."""
import ctypes as C

import numpy as np
import pytest

import s615
import workloads as W

pytestmark = pytest.mark.gpu
N = 2000
FIELDS = ("calls", "gated", "probes", "pos", "hits")


@pytest.fixture(scope="module")
def table():
    with s615.Engine(0) as eng:
        yield eng, eng.build_table(N, 16)


def key(h, n):
    a = np.stack([h[k].astype(np.uint64) for k in ("unit", "d", "e", "c4", "fp")], axis=1)
    a = a[a[:, 0] < n]
    return a[np.lexsort(a.T[::-1])]


def both_ways(table, units, flags=0):
    """(hits, counters) of the units packed on the device, checked against the host's."""
    eng, tid = table
    n = len(units)
    arr = (s615.Unit * (n + 1))(*units)
    lib = s615.lib()
    got_bytes, status = {}, {}
    # a (6,1,7) candidate with u >= B: dropped, and nothing of it is counted
    empty = s615.Unit()
    empty.cls, empty.B, empty.u, empty.w = 7, 5, 5 + 9 * 729, 5 + 117649
    assert lib.s615_unit_status(C.byref(empty)) == 1
    arr[n] = empty
    out = []
    for m in (n, n + 1):
        h, c = eng.run(tid, arr, m, flags)
        out.append((key(h, n), [getattr(c, f) for f in FIELDS]))
        b, nb = C.c_void_p(), C.c_size_t()
        s615._check(lib.s615_prepare(eng._ctx, C.cast(arr, C.c_void_p), m, C.byref(b)), "prepare")
        ni = C.c_size_t()
        lib.s615_batch_size(b, None, C.byref(ni), C.byref(nb))
        status[m], got_bytes[m] = ni.value, nb.value
        lib.s615_batch_free(eng._ctx, b)
    assert got_bytes[n] == 72 * n and got_bytes[n + 1] >= 224 * n   # which way each went
    assert status[n] == status[n + 1]                               # as many items
    np.testing.assert_array_equal(out[0][1], out[1][1])
    np.testing.assert_array_equal(out[0][0], out[1][0])
    return out[0]


def units_of(arr, n):
    return [arr[i] for i in range(n)]


@pytest.mark.parametrize("lo,hi,n", [(1000, 3000, 200), (30000, 84000, 700), (1900000, 2000000, 150)])
def test_stage1_units_and_plants(table, lo, hi, n):
    mixed = W.mixed_units(n, lo, lo, hi)
    arr, k = W.mixed_unit_array(mixed, W.plants(9, 1, lo, hi, N), W.plants234(30, 2, lo, hi, N), N)
    hits, ctr = both_ways(table, units_of(arr, k))
    assert ctr[2] > 0 and len(hits) >= 20


def test_every_class_alone_and_dropped_units(table):
    for cls in (2, 3, 4, 5):
        us = W.mixed_units(150, cls, 20000, 60000, mix={cls: 1.0})
        out = []
        for c, B, u in us:
            x = s615.Unit()
            x.cls, x.B, x.u = c, B, u
            out.append(x)
            y = s615.Unit()
            y.cls, y.B, y.u = c, u, B   # u >= B: dropped
            out.append(y)
        both_ways(table, out)
        both_ways(table, out, s615.F_SHARP)


def test_jobs_with_gaps(table):
    """Job rows of both kinds, dropped ones among them (T = 0, T >= 2^121), so that runs
    end inside, at and beyond the multiples where items start; T past 2^121 for class 5."""
    rng = np.random.RandomState(7)
    units = W.mixed_units(40, 3, 60000, 84000, mix={2: 0.3, 4: 0.7})
    jobs, nj, _ = s615.expand_units(units)
    out = []
    for i in range(min(nj, 3000)):
        j = s615.Unit.from_buffer_copy(jobs[i])
        r = rng.randint(0, 12)
        if r == 0:
            j.base[0] = j.base[1] = 0
        elif r == 1:
            j.base[1] = 1 << 57
        elif r == 2:
            j.cls = 5
        elif r == 3:
            j.cls, j.base[1] = 5, int(rng.randint(1, 2**31)) << 33
        out.append(j)
    for cut in (129, 1000, 2049, len(out)):
        both_ways(table, out[:cut])


def test_find4_units(table):
    """Class 1 as Stage-1 units, jobs and plants, and (6,1,7) find4 jobs: alone, among the
    others, with empty windows and targets at the ends of what is taken."""
    units = units_of(*s615.jobs617_band([71001, 71003], (1, 2, 3, 4)))[:1500]
    stage1 = []
    for c, B, u in W.mixed_units(120, 5, 40000, 84000, mix={1: 0.7, 4: 0.3}):
        x = s615.Unit()
        x.cls, x.B, x.u = c, B, u
        stage1.append(x)
    jobs, nj, _ = s615.expand_units(W.mixed_units(30, 6, 60000, 84000, mix={1: 0.5, 4: 0.5}))
    plants = [s615.make_plant1((a, 700, 900, 1900), lim=1999) for a in (1, 500, 699)]
    plants.append(s615.make_plant1((1, 1, 1, 1), lim=0))
    plants.append(s615.make_plant1((1, 1, 1, 1), lim=1))
    edge = []
    for T in (1, 4, 5, 64, 4 * 7**6, 4 * 7**6 + 1, 2**122 - 1, 2**122, 0):
        j = s615.Unit()
        j.cls, j.kind, j.lim, j.B, j.u = 1, 2, 1999, 83999, 5
        j.base[0], j.base[1] = T & (2**64 - 1), T >> 64
        edge.append(j)
    # lim = 1999 leaves the last targets' windows empty; the hits are those of few probes
    mixed = edge + plants + stage1 + units_of(jobs, min(nj, 900)) + units
    assert {x.cls for x in mixed} >= {1, 4, 8}
    hits, ctr = both_ways(table, mixed)
    assert ctr[2] > 0
    both_ways(table, units)
    both_ways(table, edge * 20)


def test_a_refused_unit_refuses_the_batch(table):
    eng, tid = table
    good = units_of(*W.unit_array(W.cls5_units(20000, 24000)[:200], [], N))
    for bad in (dict(cls=5, B=20005, u=8), dict(cls=2, B=40000001, u=5), dict(cls=4, B=1, u=5),
                dict(cls=1, B=20001, u=5), dict(cls=1, kind=1, B=20001, u=5, base0=12345),
                dict(cls=1, kind=1, B=20001, u=5, lim=1 << 21, base0=5489031744),
                dict(cls=8, kind=1, B=20001, u=5), dict(cls=8, B=20001, u=5, fmax1=3, fmax2=4, lim=9),
                dict(cls=8, kind=2, B=20001, u=5),
                dict(cls=3, kind=3, B=20001, u=5), dict(cls=5, kind=2, B=20001, u=5, base2=1),
                dict(cls=5, kind=1, B=20001, u=5, base0=12345)):
        x = s615.Unit()
        for k, v in bad.items():
            if k.startswith("base"):
                x.base[int(k[4])] = v
            else:
                setattr(x, k, v)
        assert s615.lib().s615_unit_status(C.byref(x)) == -3
        arr = (s615.Unit * (len(good) + 1))(*good, x)
        with pytest.raises(s615.S615Error) as e:
            eng.run(tid, arr, len(good) + 1)
        assert e.value.status == -3


def test_plain_form_of_a_device_filled_batch(table):
    eng, tid = table
    arr, n = W.unit_array(W.cls5_units(20000, 24000)[:160], [], N)
    h0, c0 = eng.run(tid, arr, n)
    h1, c1 = eng.run(tid, arr, n, s615.F_PLAIN)
    assert [getattr(c0, f) for f in FIELDS] == [getattr(c1, f) for f in FIELDS]
    np.testing.assert_array_equal(key(h0, n), key(h1, n))
