"""A graph's ranks, residual and sweep count in the batch solve do not depend on the graphs that
are solved with it: the same bits beside one small graph, among others, and in another order."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "graphchi-cpp_b200"))

pytestmark = pytest.mark.gpu

# up to 256 tiles of 128 rows a warp adds a graph's partials, beyond a block
SIZES = [1, 100, 129, 4097, 32_640, 32_768, 32_769, 33_000, 140_001, 900_001]  # the last: more tiles than warps


def build(k, n):
    import gcgpu
    s, d = gcgpu.generate_er(n, 4 * n, seed=k + 1)
    if k % 2:  # also graphs whose rows all have in-edges
        v = np.arange(n, dtype=np.uint32)
        s, d = np.concatenate([s, v]), np.concatenate([d, (v + 1) % np.uint32(n)])
    return gcgpu.Graph.from_edges(s, d, num_vertices=n, dedup=True)


@pytest.mark.parametrize("kw", [{"max_sweeps": 1}, {"max_sweeps": 3}, {"max_sweeps": 400, "tol": 1e-7}])
def test_same_bits_in_any_company(kw):
    """From initial values over 18 decades: FP64 sums of ranks that are alike are exact in any order."""
    import gcgpu
    graphs = [build(k, n) for k, n in enumerate(SIZES)]
    init = [(10.0 ** np.random.default_rng(k).uniform(-12, 6, n)).astype(np.float32) for k, n in enumerate(SIZES)]

    def solve(order):
        with gcgpu.Batch([graphs[k] for k in order]) as b:
            r, sw, res, _ = b.pagerank(init_rank=np.concatenate([init[k] for k in order]), **kw)
            return [(p.copy(), int(s), float(x)) for p, s, x in zip(b.split(r), sw, res)]
    alone = [solve([k, 1])[0] for k in range(len(graphs))]  # with one small graph only
    many = [3, 0, 6, 9, 8, 8, 2, 5, 1, 4, 7, 6, 0]
    for order in (range(len(graphs)), range(len(graphs) - 1, -1, -1), many, [7, 2]):
        for k, (ranks, sweeps, residual) in zip(order, solve(order)):
            assert np.array_equal(ranks, alone[k][0]) and (sweeps, residual) == alone[k][1:], (k, residual, alone[k][2])
    for g in graphs:
        g.free()
