"""Tables probed through their low-bit plane: the answers are the oracle's on
the same table bytes, false positives included (GPU)."""
import numpy as np
import pytest

import orc
import s615
import workloads as W
from test_gpu_cls5 import oracle_units, sorted_hits
from test_gpu_xor import random_keys

pytestmark = pytest.mark.gpu

# (N, r, layout, plane bits): every width, 4- and 8-byte and packed cells, a
# table below the first that has a plane
CASES = [
    (3000, 48, s615.LAYOUT_WIDE, 0),
    (4200, 48, s615.LAYOUT_WIDE, 8),
    (9000, 16, s615.LAYOUT_WIDE, 8),
    (9000, 15, s615.LAYOUT_PACKED, 8),
    (14501, 16, s615.LAYOUT_WIDE, 4),
    (23803, 17, s615.LAYOUT_PACKED, 2),
    (33001, 16, s615.LAYOUT_WIDE, 1),
]


def plane_bytes(m, bits):
    per = 32 // bits if bits else 1
    return (m + per - 1) // per * 4 if bits else 0


@pytest.mark.parametrize("N,r,layout,bits", CASES)
def test_query_through_plane(engine, N, r, layout, bits):
    tid = engine.build_table(N, r, layout)
    try:
        info = engine.table_info(tid)
        m = info.hdr.m_cells
        cells = ((m * r + 7) // 8 + 8 + 7) // 8 * 8 + 8 if layout == s615.LAYOUT_PACKED \
            else m * info.cell_bytes
        # one bit of 83 MB leaves the probe slow enough for the staged probe's plane too
        staged = plane_bytes(m, 4) if bits == 1 else 0
        assert info.device_bytes - cells == plane_bytes(m, bits) + staged
        t = orc.Table.from_memory(*engine.export_table(tid))
        rng = np.random.RandomState(N)
        i = rng.randint(1, N + 1, size=(2, 1 << 18)).astype(np.uint64)
        member = i[0] ** np.uint64(6) + i[1] ** np.uint64(6)
        probe = np.concatenate([member, random_keys(1 << 20, N + r), member + np.uint64(1)])
        got = engine.query(tid, probe)
        assert got[:member.size].all()
        np.testing.assert_array_equal(got, t.query(probe))
    finally:
        engine.free_table(tid)


def test_run_through_plane(engine):
    """Raw hits and counters of class-5 units, with about 2^-16 of the probes false positives."""
    N = 5600
    tid = engine.build_table(N, 16)
    try:
        assert engine.table_info(tid).device_bytes > 4 * engine.table_info(tid).hdr.m_cells
        t = orc.Table.from_memory(*engine.export_table(tid))
        units, plants = W.cls5_units(200000, 200060), W.plants(5, 3, 190000, 200060, N)
        arr, n = W.unit_array(units, plants, N)
        hits, ctr = engine.cls5_run(tid, arr, n)
        oarr, on = oracle_units(units, plants, N)
        ohits, (calls, gated, probes) = orc.cls5_run(t, oarr, on)
        assert (ctr.calls, ctr.gated, ctr.probes) == (calls, gated, probes)
        np.testing.assert_array_equal(sorted_hits(hits), sorted_hits(ohits))
    finally:
        engine.free_table(tid)


def test_plane_as_wide_as_the_cells(engine):
    """r = 8 and an 8-bit plane (a key set: the pair tables' smoke test refuses r = 8)."""
    keys = random_keys(20_000_000, 8)
    tid = engine.build_table_keys(keys, 8)
    try:
        info = engine.table_info(tid)
        m = info.hdr.m_cells
        assert info.device_bytes == 4 * m + plane_bytes(m, 8)
        t = orc.Table.from_memory(*engine.export_table(tid))
        probe = np.concatenate([keys[::16], random_keys(1 << 20, 9)])
        got = engine.query(tid, probe)
        assert got[:keys[::16].size].all()
        np.testing.assert_array_equal(got, t.query(probe))
    finally:
        engine.free_table(tid)
