"""Flag bits that s615.h does not define change nothing (GPU)."""
import numpy as np
import pytest

import s615
import workloads as W

pytestmark = pytest.mark.gpu
FIELDS = ("calls", "gated", "probes", "pos", "hits")


@pytest.mark.parametrize("bit", [8, 28, 29, 30, 31])
def test_undefined_flag_bits(engine, bit):
    N = 715
    tid = engine.build_table(N, 16)
    try:
        plants = W.plants(4, 0, 1000, 30000, N)
        for n in (40, 200):   # packed on the host, on the device
            arr, k = W.unit_array(W.cls5_units(1000, 30000)[:n], plants, N)
            h0, c0 = engine.run(tid, arr, k)
            h1, c1 = engine.run(tid, arr, k, 1 << bit)
            assert [getattr(c0, f) for f in FIELDS] == [getattr(c1, f) for f in FIELDS]
            assert c0.probes > 0 and len(h0) >= len(plants)
            np.testing.assert_array_equal(np.sort(h0, order=["unit", "fp"]),
                                          np.sort(h1, order=["unit", "fp"]))
    finally:
        engine.free_table(tid)
