"""Gauss-Seidel sweeps of wide levels, whose rows go to threads (up to 32 in-edges) and to
warps (up to 4096) where they outnumber the warps: bit for bit against sequential sums
(numpy's accumulate adds one value after another) at the edges of the classes, and not
far behind a Jacobi sweep of the same graph."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "graphchi-cpp_b200"))

pytestmark = pytest.mark.gpu

SOURCES = 5000


def wide(lengths, below, seed):
    """One row per entry of lengths, all independent: their sources are the ids below them
    (this sweep's values) or above (the sweep's before). Returns the edges, row by row."""
    rng = np.random.default_rng(seed)
    src = np.concatenate([np.sort(rng.permutation(SOURCES)[:k]) for k in lengths])
    dst = np.repeat(np.arange(len(lengths)), lengths)
    if below:
        return src.astype(np.uint32), (dst + SOURCES).astype(np.uint32)
    return (src + len(lengths)).astype(np.uint32), dst.astype(np.uint32)


def sums(lengths, x):
    """The float sums of consecutive stretches of x, each from 0 on, one value after another."""
    ends = np.cumsum(lengths)
    out = np.empty(len(lengths), np.float32)
    for k in np.unique(lengths):
        rows = np.flatnonzero(lengths == k)
        at = (ends[rows] - k)[:, None] + np.arange(k)
        vals = np.concatenate([np.zeros((len(rows), 1), np.float32), x[at]], axis=1)
        out[rows] = np.add.accumulate(vals, axis=1, dtype=np.float32)[:, -1]
    return out


CASES = {  # (row length, rows): 2368 warps sweep on 148 SMs
    "threads": [(9, 900), (31, 900), (32, 900), (8, 500), (33, 300), (1, 50)],
    "just_wide": [(16, 2369), (40, 7)],
    "just_not_wide": [(16, 2368), (40, 7)],
    "warps_few_rounds": [(33, 2000), (255, 2000), (256, 1500), (64, 700)],
    "warps_many_rounds": [(33, 9000), (100, 473), (257, 11), (32, 100)],
    "warps_past_32_rounds": [(33, 75_800), (34, 3)],
    "long_rows": [(257, 800), (511, 40), (512, 40), (513, 40), (2000, 150), (4095, 60), (4096, 60), (4097, 9), (40, 30)],
    "long_rows_many_rounds": [(257, 1500), (300, 700), (40, 9000)],
    "half_the_warps": [(300, 1184), (301, 0)],
    "half_the_warps_and_one": [(300, 1184), (301, 1)],
}


@pytest.mark.parametrize("below", [True, False])
@pytest.mark.parametrize("name", CASES)
def test_wide_levels(name, below):
    import gcgpu
    rng = np.random.default_rng(3)
    lengths = rng.permutation(np.concatenate([np.full(n, k) for k, n in CASES[name]]))
    s, d = wide(lengths, below, 4)
    rows, n = len(lengths), len(lengths) + SOURCES
    teleport, damping, sweeps = 0.15, 0.85, 2
    outdeg = np.bincount(s, minlength=n)
    od = np.maximum(outdeg, 1)
    with gcgpu.Graph.from_edges(s, d, num_vertices=n, dedup=True, out_csr=False) as g:
        got, st = g.pagerank(mode=gcgpu.PR_GS_EXACT, max_sweeps=sweeps)
        assert st.levels == (2 if below else 1)
        log = np.zeros(sweeps)
        logged, _ = g.pagerank(mode=gcgpu.PR_GS_EXACT, max_sweeps=sweeps, residuals=log)  # the tracking kernel
        edge, _ = g.pagerank(mode=gcgpu.PR_GS_EDGE, max_sweeps=sweeps)
    at = np.arange(SOURCES, n) if below else np.arange(rows)  # the rows; the others have no in-edges
    # the in-memory program: a source's value is teleport / outdeg from the first sweep on, in the sweep
    # that writes it already where the row comes later; rows feed no one
    src_val = np.where(outdeg > 0, teleport / od, teleport).astype(np.float32)
    ref = src_val.copy()
    ref[at] = (teleport + damping * sums(lengths, src_val[s]).astype(np.float64)).astype(np.float32)
    ref = np.where(outdeg > 0, ref * od.astype(np.float32), ref)
    assert np.array_equal(got, ref) and np.array_equal(logged, ref)
    # the edge-value program: the float rank over the float out-degree on the edges
    c = np.float32(teleport) / od.astype(np.float32)
    ref = np.full(n, np.float32(teleport))
    ref[at] = (teleport + damping * sums(lengths, c[s]).astype(np.float64)).astype(np.float32)
    assert np.array_equal(edge, ref)


def test_uniform_graph_keeps_up_with_jacobi():
    """4 M vertices of 16 in-edges: some forty levels of 100,000 rows, which by warps alone took
    nearly five times as long as by threads."""
    import gcgpu
    import torch
    n, m = 1 << 22, 16 << 22
    s, d = (torch.empty(m, dtype=torch.int32, device="cuda") for _ in range(2))
    gcgpu.generate_er(n, m, seed=1, src=s, dst=d)
    out = torch.empty(n, dtype=torch.float32, device="cuda")
    with gcgpu.Graph.from_edges(s, d, num_vertices=n, dedup=True, out_csr=False) as g:
        def best(**kw):
            return min(g.pagerank(max_sweeps=3, out=out, **kw)[1].device_ms for _ in range(5))
        gs, jacobi = best(mode=gcgpu.PR_GS_EXACT), best()
        assert gs < 3.5 * jacobi, (gs, jacobi)
