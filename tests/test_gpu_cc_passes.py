"""Sampled connected components at the edges of its passes: vertex counts around a warp, a
block and a grid of several vertices per thread; long chains; ids against the degrees (every
vertex's first neighbour larger than itself); a giant component whose sampled root is not its
smallest id; lists longer than one thread links. Labels are whole numbers: equal to a union-find
on the CPU."""
import os
import sys

import numpy as np
import pytest
from scipy.sparse import coo_matrix
from scipy.sparse.csgraph import connected_components

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "graphchi-cpp_b200"))

pytestmark = pytest.mark.gpu


def labels(n, s, d):
    """The smallest id of each vertex's component."""
    _, comp = connected_components(coo_matrix((np.ones(len(s)), (s, d)), shape=(n, n)), directed=False)
    first = np.full(comp.max() + 1, n, np.int64)
    np.minimum.at(first, comp, np.arange(n))
    return first[comp]


def make(kind, n):
    rng = np.random.default_rng(n)
    if kind == "sparse":
        return rng.integers(0, n, n // 2 + 1), rng.integers(0, n, n // 2 + 1)
    if kind == "dense":
        return rng.integers(0, n, 4 * n), rng.integers(0, n, 4 * n)
    if kind == "chain":  # in id order
        return np.arange(n - 1), np.arange(1, n)
    if kind == "shuffled chain":
        p = rng.permutation(n)
        return p[:-1], p[1:]
    if kind == "star":  # around the last vertex
        return np.arange(n - 1), np.full(n - 1, n - 1)
    if kind == "low tail":  # ids below n / 2 in a chain joined to the rest's star by one edge
        h = n // 2
        return (np.concatenate([np.arange(h - 1), np.full(n - h - 1, h), [h - 1]]),
                np.concatenate([np.arange(1, h), np.arange(h + 1, n), [n - 1]]))
    assert kind == "lists"  # stars of 60..70 leaves, none of them the giant
    hubs = np.repeat(np.arange(11) * 80, 60 + np.arange(11))
    leaf = np.concatenate([80 * i + 1 + np.arange(60 + i) for i in range(11)])
    rest = np.arange(1000, n - 1)
    return np.concatenate([leaf, rest]), np.concatenate([hubs, rest + 1])


CASES = [(k, n) for k in ("sparse", "dense", "star") for n in (2, 31, 32, 33, 255, 256, 257, 1025)]
CASES += [(k, n) for k in ("sparse", "dense", "chain", "shuffled chain", "star", "low tail", "lists")
          for n in (8193, 303104 * 4 + 33)]


@pytest.mark.parametrize("symmetrise", [True, False])
@pytest.mark.parametrize("kind,n", CASES)
def test_labels(kind, n, symmetrise):
    import gcgpu
    s, d = (x.astype(np.uint32) for x in make(kind, n))
    with gcgpu.Graph.from_edges(s, d, num_vertices=n, dedup=True, symmetrise=symmetrise) as g:
        got, st = g.connected_components()
    ref = labels(n, s, d)
    assert st.passes == 2
    assert np.array_equal(got, ref)
    assert st.ncomponents == np.count_nonzero(ref == np.arange(n))
