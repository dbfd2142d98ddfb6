"""Batched personalised PageRank at the edges of its layouts (widths around one lane
group, one slice and several) and of its segments (rows of 255..257, 511..513 and many
in-edges), against the oracle at fixed sweeps and against single-source solves."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "graphchi-cpp_b200"))
sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))

pytestmark = pytest.mark.gpu

N = 4000


@pytest.fixture(scope="module")
def edges():
    rng = np.random.default_rng(3)
    src, dst = [rng.integers(0, N, 6 * N)], [rng.integers(0, N, 6 * N)]
    for i, k in enumerate([255, 256, 257, 511, 512, 513, 2049, 3900]):
        src.append(rng.choice(N, size=k, replace=False))
        dst.append(np.full(k, 11 + 7 * i))
    return np.concatenate(src).astype(np.uint32), np.concatenate(dst).astype(np.uint32)


@pytest.mark.parametrize("k", [1, 7, 8, 9, 32, 33, 63, 64, 65, 96, 97, 130, 256, 257])
def test_widths_vs_oracle(edges, k):
    import gcgpu
    import oracle as O
    s, d = edges
    go = O.OracleGraph(s, d)
    sources = np.random.default_rng(k).integers(0, N, k).astype(np.uint32)
    with gcgpu.Graph.from_edges(s, d, dedup=True, out_csr=False) as g:
        got, st = g.ppr_batched(sources, max_sweeps=9, teleport=0.15)
        ref, _ = go.ppr(sources, damping=0.85, max_sweeps=9, tol=0.0)
        assert st.sweeps == 9
        assert float(np.abs(got - ref).sum(axis=0).max()) <= 1e-6
        # to a tolerance: columns retire one by one and the matrix is compacted
        got, _ = g.ppr_batched(sources, max_sweeps=500, teleport=0.15, tol=1e-8)
        for j in sorted({0, k // 2, k - 1}):
            one, _ = g.pagerank(max_sweeps=500, teleport=0.15, tol=1e-8, source=int(sources[j]))
            assert np.abs(got[:, j] - one).sum() <= 1e-6
