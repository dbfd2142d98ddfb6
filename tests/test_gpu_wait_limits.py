"""The bounded waits of the cooperative PageRank launches: a barrier that waits for an arrival that
does not come ends the call with GCG_ERR_TIMEOUT, and the graph solves as before afterwards."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "graphchi-cpp_b200"))

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [
    {"max_sweeps": 5}, {"max_sweeps": 100, "tol": 1e-6},
    {"mode": 1, "max_sweeps": 3}, {"mode": 1, "max_sweeps": 20, "tol": 1e-6}, {"mode": 3, "max_sweeps": 10}],
    ids=["one_launch", "one_launch_tol", "gs", "gs_tol", "gs_edge"])
@pytest.mark.parametrize("scale", [4, 14])
def test_a_missing_arrival_times_out(kw, scale):
    import gcgpu
    assert (gcgpu.PR_GS_EXACT, gcgpu.PR_GS_EDGE) == (1, 3)
    s, d = gcgpu.generate_rmat(scale, 16 << scale, seed=3)
    with gcgpu.Graph.from_edges(s, d, dedup=True, out_csr=False) as g:
        ref, st = g.pagerank(**kw)
        for _ in range(3):
            with pytest.raises(gcgpu.GcgError) as e:
                g.pagerank(flags=gcgpu.PR_TEST_BARRIER_TIMEOUT, **kw)
            assert gcgpu.STATUS_NAMES[e.value.status] == "GCG_ERR_TIMEOUT"
            r, again = g.pagerank(**kw)
            assert np.array_equal(r, ref) and again.sweeps == st.sweeps
