"""Components of graphs with fewer neighbours than vertices, where the sample also decides by its
vertices' neighbours whether a second round can find a giant component: uniform graphs below and
above that, a dense core among isolated vertices, chains and stars, at both sides of the line."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "graphchi-cpp_b200"))

pytestmark = pytest.mark.gpu


def labels(n, s, d):
    """The smallest id of each vertex's component (scipy's components, relabelled)."""
    from scipy.sparse import coo_matrix
    from scipy.sparse.csgraph import connected_components
    _, comp = connected_components(coo_matrix((np.ones(len(s), np.int8), (s, d)), shape=(n, n)), directed=False)
    least = np.full(comp.max() + 1, n)
    np.minimum.at(least, comp, np.arange(n))
    return least[comp].astype(np.uint32)


def edges(name, rng):
    if name.startswith("uniform_"):
        m = int(name[8:])
        return 200_000, rng.integers(0, 200_000, m), rng.integers(0, 200_000, m)
    if name == "core":
        ids = rng.permutation(400_000)[:20_000]
        return 400_000, ids[rng.integers(0, 20_000, 150_000)], ids[rng.integers(0, 20_000, 150_000)]
    if name == "chain":
        p = rng.permutation(300_000)[:100_000]
        return 300_000, p[:-1], p[1:]
    if name == "line":  # neighbours = vertices (symmetrised): the path of n / 2 + 1 vertices
        return 100_000, np.arange(50_000), np.arange(1, 50_001)
    if name == "line_and_one":
        return 100_000, np.arange(50_001), np.arange(1, 50_002)
    hub = 299_999 if name == "star_high" else 0
    leaves = rng.permutation(299_000)[:50_000] + 1
    return 300_000, leaves, np.full(50_000, hub)


@pytest.mark.parametrize("symmetrise", [True, False])
@pytest.mark.parametrize("name", ["uniform_0", "uniform_1", "uniform_20000", "uniform_90000", "uniform_100000",
                                  "uniform_130000", "uniform_250000", "core", "chain", "line", "line_and_one",
                                  "star_low", "star_high"])
def test_labels(name, symmetrise):
    import gcgpu
    n, s, d = edges(name, np.random.default_rng(7))
    with gcgpu.Graph.from_edges(s.astype(np.uint32), d.astype(np.uint32), num_vertices=n, dedup=True,
                                symmetrise=symmetrise) as g:
        ref = labels(n, s, d)
        for _ in range(3):
            got, st = g.connected_components()
            assert np.array_equal(got, ref) and st.ncomponents == len(np.unique(ref))
