"""The staged probe against the oracle, in the checked build, and the large batches that do
not go through it (GPU).  Run as a script it is the checked build's child process."""
import json
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
N, R = 28000, 16


def units():
    import workloads as W
    return W.cls5_units(1150000, 1150400)[:700], W.plants(3, 6, 1100000, 1170000, N)


@pytest.mark.gpu
def test_staged_hits_are_the_oracles(engine):
    import numpy as np
    import orc
    import s615
    import workloads as W
    from test_gpu_cls5 import oracle_units, sorted_hits
    us, plants = units()
    arr, n = W.unit_array(us, plants, N)
    tid = engine.build_table(N, R)
    try:
        before = engine.launches
        hits, ctr = engine.cls5_run(tid, arr, n)
        assert engine.launches - before >= 5     # emit, the steps, resolve
        t = orc.Table.from_memory(*engine.export_table(tid))
        oarr, on = oracle_units(us, plants, N)
        ohits, (calls, gated, probes) = orc.cls5_run(t, oarr, on)
        assert probes > 2.5e7 and len(ohits) > 300
        assert (ctr.calls, ctr.gated, ctr.probes) == (calls, gated, probes)
        np.testing.assert_array_equal(sorted_hits(hits), sorted_hits(ohits))
        before = engine.launches                 # the sharper gate's kernel has no stages
        engine.cls5_run(tid, arr, n, s615.F_SHARP)
        assert engine.launches - before <= 4
    finally:
        engine.free_table(tid)


@pytest.mark.gpu
@pytest.mark.parametrize("r,shards", [(15, 1), (20, 2)])
def test_probed_directly(engine, r, shards):
    """Tables of fewer than 16 bits, and shard sets, have no planes for the stages."""
    import workloads as W
    us, plants = units()
    arr, n = W.unit_array(us, plants, N)
    tid = engine.build_table(N, r) if shards == 1 else engine.build_table_sharded(N, r, shards)
    try:
        before = engine.launches
        hits, ctr = engine.cls5_run(tid, arr, n)
        assert engine.launches - before <= 4
        assert ctr.probes > 2.5e7
        for j, p in enumerate(plants):
            assert ((hits["unit"] == len(us) + j) & (hits["fp"] == p.fp)).any()
    finally:
        engine.free_table(tid)


def child():
    sys.path[:0] = [os.path.join(ROOT, "six-one-five_b200"), HERE]
    import s615
    import workloads as W
    with s615.Engine(0) as eng:
        tid = eng.build_table(N, R)
        arr, n = W.unit_array(*units(), N)
        before = eng.launches
        h, c = eng.cls5_run(tid, arr, n)
        rows = sorted((int(x["unit"]), int(x["d"]), int(x["e"]), int(x["fp"])) for x in h)
        print(json.dumps({"checked": s615.lib().s615_checked_build(), "flags": eng.check_flags(),
                          "launches": eng.launches - before, "probes": c.probes,
                          "plants": len({x[0] for x in rows if x[0] >= n - 3})}))


@pytest.mark.gpu
def test_checked_build_sets_no_flag_in_the_stages():
    p = subprocess.run([sys.executable, os.path.abspath(__file__)], env=dict(os.environ, S615_CHECKED="1"),
                       capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stdout[-2000:] + p.stderr[-4000:]
    got = json.loads(p.stdout.strip().splitlines()[-1])
    assert got["checked"] == 1 and got["flags"] == 0
    assert got["launches"] >= 5 and got["probes"] > 2.5e7 and got["plants"] == 3


if __name__ == "__main__":
    child()
