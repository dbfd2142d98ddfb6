"""The autotuner's choice includes the one-launch solve that small graphs get by default."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "graphchi-cpp_b200"))

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("configured", [False, True])
def test_autotuned_small_graph_keeps_the_one_launch_solve(configured):
    """16 edges a vertex, 2^16 vertices: the one launch takes half the queued kernels' time."""
    import gcgpu
    s, d = gcgpu.generate_rmat(16, 16 << 16, seed=2)
    with gcgpu.Graph.from_edges(s, d, dedup=True, out_csr=False) as g:
        ref, st = g.pagerank(max_sweeps=5)
        assert st.kernel_launches == 1
        if configured:  # by hand: the queued kernels
            g.pagerank_config(16384, 2)
            assert g.pagerank(max_sweeps=5)[1].kernel_launches > 1
        hub, run, ms = g.pagerank_autotune(sweeps=8)
        assert g.pagerank_config() == (hub, run) and g.pagerank_tiers() == 1 and ms > 0
        r, st = g.pagerank(max_sweeps=5)
        assert st.kernel_launches == 1 and np.array_equal(r, ref)


def test_refused_autotune_changes_nothing():
    import gcgpu
    s, d = gcgpu.generate_rmat(13, 9 << 13, seed=4)
    with gcgpu.Graph.from_edges(s, d, dedup=True, out_csr=False) as g:
        with pytest.raises(gcgpu.GcgError):
            g.pagerank_autotune(sweeps=0)
        assert g.pagerank(max_sweeps=5)[1].kernel_launches == 1
