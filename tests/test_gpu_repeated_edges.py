"""The sharder on edge lists with many repeats of few edges: out-degrees counted from runs of
one source, repeats taken off run by run, against numpy; and no slower for it."""
import os
import sys
import time

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "graphchi-cpp_b200"))

pytestmark = pytest.mark.gpu


def check(s, d, n, dedup):
    import gcgpu
    with gcgpu.Graph.from_edges(s, d, num_vertices=n, dedup=dedup, out_csr=False) as g:
        deg = g.degrees()
        rp, col = g.csr()
    keep = s != d
    keys = d[keep].astype(np.int64) * n + s[keep]
    keys = np.unique(keys) if dedup else np.sort(keys)
    assert np.array_equal(deg[:, 0], np.bincount(keys // n, minlength=n))
    assert np.array_equal(deg[:, 1], np.bincount(keys % n, minlength=n))
    assert np.array_equal(rp, np.concatenate([[0], np.cumsum(np.bincount(keys // n, minlength=n))]))
    assert np.array_equal(col, (keys % n).astype(np.uint32))


@pytest.mark.parametrize("dedup", [True, False])
@pytest.mark.parametrize("n", [2, 3, 20, 200, 256, 300])
def test_random_repeats(n, dedup):
    rng = np.random.default_rng(n)
    s, d = (rng.integers(0, n, 200_003).astype(np.uint32) for _ in range(2))
    check(s, d, n, dedup)


@pytest.mark.parametrize("dedup", [True, False])
@pytest.mark.parametrize("runs", [  # copies of edge 0, 1, ..: around a window of 32 and a warp's share of 256 and 512
    [1], [2], [31], [32], [33], [64], [65], [255], [256], [257], [511], [512], [513], [1025],
    [31, 1, 32, 33], [1, 32, 31], [64, 64, 64], [512, 512, 1], [7, 505, 512, 3], [100] * 11, [1] * 700 + [700]])
def test_runs_at_window_edges(runs, dedup):
    k = np.arange(len(runs))
    s = np.repeat(k % 13, runs).astype(np.uint32)           # a few sources, each in many runs
    d = np.repeat(13 + k // 13, runs).astype(np.uint32)
    check(s, d, 13 + len(runs) // 13 + 1, dedup)


def test_self_loops_between_runs():
    rng = np.random.default_rng(1)
    s = np.repeat(rng.integers(0, 8, 3000), rng.integers(1, 60, 3000)).astype(np.uint32)
    d = np.repeat(rng.integers(0, 8, 500), 400)[: len(s)].astype(np.uint32)
    s = s[: len(d)]
    for dedup in (True, False):
        check(s, d, 8, dedup)


@pytest.mark.parametrize("n", [20, 200])
def test_no_slower_than_with_out_lists(n):
    """16 M edges among few vertices: an atomic per repeat took 7 and 17 times as long as the build
    that makes the out-lists too."""
    import gcgpu
    import torch
    s, d = (torch.empty(16 << 20, dtype=torch.int32, device="cuda") for _ in range(2))
    gcgpu.generate_er(n, 16 << 20, seed=1, src=s, dst=d)

    def best(out_csr):
        t = []
        for _ in range(6):
            t0 = time.perf_counter()
            gcgpu.Graph.from_edges(s, d, num_vertices=n, dedup=True, out_csr=out_csr).free()
            t.append(time.perf_counter() - t0)
        return min(t)
    one, both = best(False), best(True)
    assert one < 2 * both, (one, both)
