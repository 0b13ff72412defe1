"""s615_verify gives every hit's pairs whether few hits share the GPU (many warps to
a hit) or many do (one warp each) (GPU)."""
import numpy as np
import pytest

import s615
import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 40, 300])
@pytest.mark.parametrize("N", [3, 40, 76667])
def test_pairs_for_few_and_many_hits(engine, N, copies):
    plants = [W.Plant(3200003, 6 * (i + 1), 17 + i, 5 + 2 * i, min(a, b), max(a, b))
              for i, (a, b) in enumerate([(1, 2), (1, N), (2, N), (N - 1, N), (N // 2, N // 2 + 1),
                                          (1, N - 1), (max(1, N // 3), N), (N // 2 + 1, N)])
              if a != b]
    arr, n = W.unit_array([], plants, N)
    hits = np.zeros(n * copies, dtype=s615.HIT_DTYPE)
    for j in range(copies):
        for i, p in enumerate(plants):
            hits[j * n + i] = (i, 0, 0, p.d, p.e, 0, p.fp)
    sols = engine.verify(arr, n, hits, N, cap=8 * len(hits))
    got = sorted((s.unit, s.d, s.e, s.c1, s.c2) for s in sols)
    want = sorted((i, p.d, p.e, p.c1, p.c2) for i, p in enumerate(plants))
    assert got == sorted(want * copies)
