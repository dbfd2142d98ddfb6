"""The one-launch solve of small graphs against the queued sweep kernels: the same
chunks, sums and order, so the ranks are the same bits; the FP64 residuals are
added in another order."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "graphchi-cpp_b200"))

pytestmark = pytest.mark.gpu


def star(n):
    """Vertex 0 gathers from everyone (one row over many CTAs) and feeds a ring."""
    v = np.arange(1, n, dtype=np.uint32)
    return np.concatenate([v, v]), np.concatenate([np.zeros(n - 1, np.uint32), np.roll(v, 1)])


def graph_edges(name):
    import gcgpu
    if name == "one_edge":
        return np.array([1], np.uint32), np.array([0], np.uint32)
    if name == "one_chunk_and_one":  # 257 edges into one row
        return np.arange(1, 258, dtype=np.uint32), np.zeros(257, np.uint32)
    if name == "stars":
        s, d = star(300_001)
        s2, d2 = star(70_000)
        return np.concatenate([s, s2]), np.concatenate([d, d2 + 150_000])
    if name == "rmat13":
        return gcgpu.generate_rmat(13, 9 << 13, seed=4)
    if name == "rmat18_odd":
        s, d = gcgpu.generate_rmat(18, 1_999_999, seed=5)
        return s % 200_003, d % 200_003
    return gcgpu.generate_er(50_021, 400_003, seed=6)


def both(g, **kw):
    """The solve in one launch, then by the queued kernels (which a launch configuration
    set by hand selects)."""
    a, sa = g.pagerank(**kw)
    assert sa.kernel_launches == 1
    g.pagerank_config(*g.pagerank_config())
    b, sb = g.pagerank(**kw)
    assert sb.kernel_launches > 1
    return a, sa, b, sb


@pytest.mark.parametrize("sweeps,tol", [(1, 0.0), (2, 0.0), (7, 0.0), (1000, 1e-8)])
@pytest.mark.parametrize("name", ["one_edge", "one_chunk_and_one", "stars", "rmat13", "rmat18_odd", "er"])
def test_same_bits_as_queued_kernels(name, sweeps, tol):
    import gcgpu
    s, d = graph_edges(name)
    with gcgpu.Graph.from_edges(s, d, dedup=True, out_csr=False) as g:
        a, sa, b, sb = both(g, max_sweeps=sweeps, tol=tol)
        assert np.array_equal(a, b)
        assert (sa.sweeps, sa.converged) == (sb.sweeps, sb.converged)
        assert np.isclose(sa.residual, sb.residual, rtol=1e-10, atol=1e-300)


@pytest.mark.parametrize("form", ["init_rank", "init_rank_device", "source", "source_without_in_edges", "logs"])
def test_forms_of_the_call(form):
    import gcgpu
    import torch
    s, d = graph_edges("rmat13")
    with gcgpu.Graph.from_edges(s, d, dedup=True, out_csr=False) as g:
        n = g.num_vertices
        indeg = g.degrees()[:, 0]
        kw = {"max_sweeps": 12}
        logs = []
        if form.startswith("init_rank"):
            init = np.random.default_rng(1).uniform(0.1, 3.0, n).astype(np.float32)
            kw["init_rank"] = torch.from_numpy(init).cuda() if form.endswith("device") else init
        elif form == "source":
            kw["source"] = int(np.argmax(indeg))
        elif form == "source_without_in_edges":
            kw["source"] = int(np.flatnonzero(indeg == 0)[0])
        else:
            logs = [(np.zeros(12), np.zeros(12), np.zeros(24, np.uint64)) for _ in range(2)]
            kw.update(residuals=logs[0][0], delta_log=logs[0][1], work_log=logs[0][2])
        a, sa = g.pagerank(**kw)
        assert sa.kernel_launches == 1
        if logs:
            kw.update(residuals=logs[1][0], delta_log=logs[1][1], work_log=logs[1][2])
        g.pagerank_config(*g.pagerank_config())
        b, sb = g.pagerank(**kw)
        assert np.array_equal(a, b) and sa.sweeps == sb.sweeps == 12
        for x, y in zip(*logs) if logs else []:
            assert np.allclose(x.astype(np.float64), y.astype(np.float64), rtol=1e-10, atol=0)


def test_output_over_the_initial_vector():
    import gcgpu
    import torch
    s, d = graph_edges("rmat13")
    with gcgpu.Graph.from_edges(s, d, dedup=True, out_csr=False) as g:
        init = np.random.default_rng(2).uniform(0.1, 3.0, g.num_vertices).astype(np.float32)
        ref, _ = g.pagerank(max_sweeps=5, init_rank=init)
        v = torch.from_numpy(init).cuda()
        g.pagerank(max_sweeps=5, init_rank=v, out=v)
        assert np.array_equal(v.cpu().numpy(), ref)
