"""Triangle counts where the counting kernel changes its ways: fewer and more vertices
than it has bits for (16,384 ranks), neighbours below those ranks (the hashed filter and
the search behind it), one vertex with more edges than a task, lists around 32, 64 and
192 candidates, repeated edges, no triangles. Against the oracle: total, per-rank counts
and ranking."""
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


def case(name):
    rng = np.random.default_rng(5)
    if name == "triangle":
        return np.array([0, 1, 2]), np.array([1, 2, 0])
    if name == "path":
        return np.arange(999), np.arange(1, 1000)
    if name == "cliques_33_65_97_193_257":  # candidate lists of every length up to 255
        out, at = [], 0
        for k in (33, 65, 97, 193, 257):
            out.append(clique(np.arange(at, at + k)))
            at += k
        return tuple(np.concatenate(x) for x in zip(*out))
    if name == "uniform_dense":  # 40,000 vertices of degree ~60: most are below the top ranks
        return rng.integers(0, 40000, 1200000), rng.integers(0, 40000, 1200000)
    if name == "uniform_16385":
        return rng.integers(0, 16385, 300000), rng.integers(0, 16385, 300000)
    if name == "uniform_16384":
        return rng.integers(0, 16384, 300000), rng.integers(0, 16384, 300000)
    if name == "wheel":  # a hub of 30,000 over a ring: its edges are many tasks
        r = np.arange(1, 30001)
        return np.concatenate([r, r]), np.concatenate([np.zeros(30000, int), np.roll(r, 1)])
    if name == "low_cliques":  # cliques of 20 below 20,000 vertices of higher degree
        s, d = [], []
        for c in range(300):
            x, y = clique(np.arange(c * 20, c * 20 + 20))
            s.append(x), d.append(y)
        s.append(rng.integers(6000, 26000, 400000)), d.append(rng.integers(6000, 26000, 400000))
        return np.concatenate(s), np.concatenate(d)
    import gcgpu
    s, d = gcgpu.generate_rmat(17, 20 << 17, seed=8)
    return s % 100003, d % 100003


@pytest.mark.parametrize("symmetrise", [True, False])
@pytest.mark.parametrize("name", ["triangle", "path", "cliques_33_65_97_193_257", "uniform_dense", "uniform_16384",
                                  "uniform_16385", "wheel", "low_cliques", "rmat17_folded"])
def test_counts_vs_oracle(name, symmetrise):
    import gcgpu
    import oracle as O
    s, d = (x.astype(np.uint32) for x in case(name))
    if symmetrise:
        go = O.OracleGraph(np.concatenate([s, d]), np.concatenate([d, s]))
    else:
        go = O.OracleGraph(s, d)
    ref, per_ref, map_ref = go.tc()
    with gcgpu.Graph.from_edges(s, d, dedup=True, symmetrise=symmetrise) as g:
        total, per, vmap, st = g.triangle_count()
        assert total == ref == st.triangles
        assert np.array_equal(vmap, map_ref)
        assert np.array_equal(per, per_ref)
