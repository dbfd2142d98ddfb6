"""The sharder's row pointers where many rows are empty: gaps around the length from which a
warp fills them together, before the first key, between keys and after the last one."""
import os
import sys
import time

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "graphchi-cpp_b200"))

pytestmark = pytest.mark.gpu


def check(rows, repeat, n, dedup):
    import gcgpu
    d = np.repeat(rows, repeat).astype(np.uint32)
    s = np.where(d == 0, 1, 0).astype(np.uint32) + np.arange(len(d), dtype=np.uint32) % np.uint32(2)
    with gcgpu.Graph.from_edges(s, d, num_vertices=n, dedup=dedup, out_csr=False) as g:
        rp, col = g.csr()
    keys = d.astype(np.int64) * n + s
    keys = keys[s != d]
    keys = np.unique(keys) if dedup else np.sort(keys)
    assert np.array_equal(rp, np.concatenate([[0], np.cumsum(np.bincount(keys // n, minlength=n))]))
    assert np.array_equal(col, (keys % n).astype(np.uint32))


@pytest.mark.parametrize("dedup", [True, False])
@pytest.mark.parametrize("gap", [1, 2, 31, 32, 33, 34, 63, 64, 65, 1000])
@pytest.mark.parametrize("after", [0, 1, 31, 32, 33, 1000])
def test_gaps(gap, after, dedup):
    for first in (0, 1, 31, 32, 33, 34, 500):
        rows = first + gap * np.arange(40)
        for repeat in (1, 3):  # four rows per key divide the two kernels
            check(rows, repeat, int(rows[-1]) + 1 + after, dedup)


@pytest.mark.parametrize("dedup", [True, False])
def test_random_gaps_over_many_windows(dedup):
    rng = np.random.default_rng(2)
    rows = np.cumsum(rng.choice([1, 1, 1, 2, 31, 32, 33, 34, 300], 20_000))
    check(rows, rng.integers(1, 4, len(rows)), int(rows[-1]) + 77, dedup)


def test_a_thousand_edges_among_32m_vertices():
    """By the threads of the 1,000 keys alone the rows took 20 ms."""
    import gcgpu
    n = 1 << 25
    s, d = gcgpu.generate_er(n, 1000, seed=1)
    best = 1e9
    for _ in range(4):
        t0 = time.perf_counter()
        g = gcgpu.Graph.from_edges(s, d, num_vertices=n, dedup=True, out_csr=False)
        best = min(best, time.perf_counter() - t0)
        rp, _ = g.csr()
        g.free()
    assert np.array_equal(rp[1:], np.cumsum(np.bincount(d[s != d], minlength=n)))
    assert best < 8e-3, best
