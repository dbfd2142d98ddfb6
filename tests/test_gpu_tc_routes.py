"""Triangle counts by each of the three ways that the degrees choose: short lists (searched edge by
edge), long lists of vertices of like degree (grouped, the low candidates in pairs), and skewed
degrees (grouped). Against the oracle: total, per-rank counts and ranking."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "graphchi-cpp_b200"))
sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "oracle"))

pytestmark = pytest.mark.gpu


def clique(ids):
    i, j = np.triu_indices(len(ids), 1)
    return ids[i], ids[j]


def uniform(rng, n, degree):
    return rng.integers(0, n, n * degree // 2), rng.integers(0, n, n * degree // 2)


def joined(*parts):
    return tuple(np.concatenate(x) for x in zip(*parts))


def case(name):
    """The edges, and whether the mean degree of an edge's end is below 96 (short lists) and, where
    not, below four times the mean degree (flat)."""
    rng = np.random.default_rng(6)
    if name == "short_uniform":
        return uniform(rng, 30_000, 40), True, None
    if name == "short_with_a_clique":  # lists that are merged, batches dealt out one by one
        return joined(uniform(rng, 200_000, 8), clique(np.arange(0, 199_000, 1500))), True, None
    if name == "short_stars":
        hubs = [(np.full(90, h), 1000 + 90 * h + np.arange(90)) for h in range(300)]
        return joined(*hubs, uniform(rng, 28_000, 4)), True, None
    if name.startswith("flat_uniform_"):  # the top 16,384 ranks have a bit each
        return uniform(rng, int(name[13:]), 120), False, True
    if name == "flat_communities":  # most candidates below the top ranks are triangles
        parts = []
        for c in range(200):
            s, d = uniform(rng, 150, 300)
            parts.append((s + 150 * c, d + 150 * c))
        return joined(*parts), False, True
    if name == "flat_cliques":  # around the number of low elements from which pairs are searched
        at, parts = 0, []
        for k in [100, 101, 127, 128, 129, 130, 131, 132, 133, 160, 161, 192, 193] * 12:
            parts.append(clique(np.arange(at, at + k)))
            at += k
        return joined(*parts), False, True
    if name == "skewed":  # hubs over a graph whose vertices are mostly below the top ranks
        hubs = [(np.full(5000, h), rng.integers(0, 40_000, 5000)) for h in range(60)]
        return joined(*hubs, uniform(rng, 40_000, 60)), False, False
    hubs = [(np.full(9000, h), rng.integers(0, 60_000, 9000)) for h in range(60)]
    parts = []
    for c in range(300):
        s, d = uniform(rng, 150, 90)
        parts.append((s + 150 * c, d + 150 * c))
    return joined(*hubs, *parts), False, False


@pytest.mark.parametrize("symmetrise", [True, False])
@pytest.mark.parametrize("name", ["short_uniform", "short_with_a_clique", "short_stars", "flat_uniform_16384",
                                  "flat_uniform_16385", "flat_uniform_40000", "flat_communities", "flat_cliques",
                                  "skewed", "skewed_communities"])
def test_counts_vs_oracle(name, symmetrise):
    import gcgpu
    import oracle as O
    (s, d), short, flat = case(name)
    s, d = s.astype(np.uint32), d.astype(np.uint32)
    go = O.OracleGraph(*((np.concatenate([s, d]), np.concatenate([d, s])) if symmetrise else (s, d)))
    ref, per_ref, map_ref = go.tc()
    with gcgpu.Graph.from_edges(s, d, dedup=True, symmetrise=symmetrise) as g:
        deg = g.degrees().sum(axis=1).astype(np.float64) / (2 if symmetrise else 1)
        edge_degree = (deg ** 2).sum() / deg.sum()
        assert (edge_degree < 96) == short
        if not short:
            assert (edge_degree < 4 * deg.mean()) == flat
        total, per, vmap, st = g.triangle_count()
        assert total == ref == st.triangles
        assert np.array_equal(vmap, map_ref)
        assert np.array_equal(per, per_ref)
