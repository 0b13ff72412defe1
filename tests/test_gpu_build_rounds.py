"""Table builder: peel rounds that go out in batches (GPU)."""
import numpy as np
import pytest

import s615

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [5880, 5950, 9000])
def test_device_build_rounds_in_batches(engine, N):
    # Peel rounds of up to 2^21 candidates go out several at a time with their
    # sizes on the device.  0.097 m cells are the second round's candidates:
    # 2.07 million at N = 5,880 (batched from round 2), 2.12 million at 5,950
    # (from round 3), 4.8 million at 9,000.  Under a budget of
    # 11.65 bytes per N^2 there is no room for the claimed-cell list, and every
    # round scans all cells: the same bytes.
    r = 20
    tid = engine.build_table(N, r)
    try:
        h0, p0 = engine.export_table(tid)
    finally:
        engine.free_table(tid)
    with s615.Engine(0, hbm_budget=int((100 << 20) * (N / 3000) ** 2)) as tight:
        t2 = tight.build_table(N, r)
        h1, p1 = tight.export_table(t2)
    assert bytes(h0) == bytes(h1)
    np.testing.assert_array_equal(p0, p1)
