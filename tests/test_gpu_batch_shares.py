"""The batch solve's vertex phase at the edges of its shares: graphs around one 128-row tile and
several, without edges or without vertices in between, fewer tiles than warps and more, and graphs
that leave early. Each graph's ranks are the bits of its own solve at fixed sweeps, and its residual
the FP64 sum of the same terms in another order."""
import numpy as np
import pytest

import gcgpu

pytestmark = pytest.mark.gpu


def ring(n, extra, seed):
    """n vertices that all have in-edges (a ring), plus random edges."""
    rng = np.random.default_rng(seed)
    v = np.arange(n)
    return (np.concatenate([v, rng.integers(0, n, extra)]).astype(np.uint32),
            np.concatenate([(v + 1) % n, rng.integers(0, n, extra)]).astype(np.uint32))


SIZES = {
    "few tiles": [2, 127, 128, 129, 0, 3, 255, 256, 257],
    "no edges first and last": [0, 0, 129, 0, 4097, 0, 0],
    "more tiles than warps": [700001, 1, 128 * 37, 2, 50021],
    "many graphs": [2 + 37 * k % 300 for k in range(1024)],
}


@pytest.mark.parametrize("name", SIZES)
def test_shares(name):
    graphs = []
    for k, n in enumerate(SIZES[name]):
        s, d = ring(n, 3 * n, k) if n > 1 else (np.zeros(0, np.uint32),) * 2
        graphs.append(gcgpu.Graph.from_edges(s, d, num_vertices=max(n, 1), dedup=True))
    with gcgpu.Batch(graphs) as b:
        r, sw, res, _ = b.pagerank(max_sweeps=5, tol=0.0)
        rt, swt, rest, _ = b.pagerank(max_sweeps=300, tol=1e-6)
        for k, (g, part, part_t) in enumerate(zip(graphs, b.split(r), b.split(rt))):
            if len(graphs) > 64 and k % 41:
                continue
            own, st = g.pagerank(max_sweeps=5, tol=0.0)
            assert np.array_equal(part, own), k
            assert abs(res[k] - st.residual) <= 1e-12 * max(st.residual, 1e-300), k
            own, _ = g.pagerank(max_sweeps=int(swt[k]), tol=0.0)
            assert np.array_equal(part_t, own) and rest[k] <= 1e-6, k
    for g in graphs:
        g.free()
