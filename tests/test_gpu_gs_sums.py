"""The Gauss-Seidel sweep's parallel evaluation of sequential float sums, bit for bit
against a sequential restatement (numpy's accumulate adds one value after another):
row lengths at the edges of the thread, warp and block classes and of the steps, and
values that make ties, zeros, subnormals, negatives, infinities and NaN."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "graphchi-cpp_b200"))

pytestmark = pytest.mark.gpu

LENGTHS = [1, 8, 9, 31, 32, 33, 255, 256, 257, 319, 320, 321, 1023, 1024, 1025, 1089, 2048, 2049, 3500, 5800]
N = 6000


def rows_graph(seed):
    """Rows of the given lengths at ids spread over the range (some before, some after
    their sources in the visit order), plus thin random edges."""
    rng = np.random.default_rng(seed)
    src, dst = [], []
    for i, k in enumerate(LENGTHS * 2):
        v = 37 + i * 149
        u = rng.choice(np.setdiff1d(np.arange(N), [v]), size=k, replace=False)
        src.append(u)
        dst.append(np.full(k, v))
    src.append(rng.integers(0, N, 4 * N))
    dst.append(rng.integers(0, N, 4 * N))
    return np.concatenate(src).astype(np.uint32), np.concatenate(dst).astype(np.uint32)


def restated(rp, col, outdeg, sweeps, teleport, damping):
    """The in-memory program (pagerank.cpp:121-146) with any constants."""
    od = outdeg.astype(np.float32)
    with np.errstate(all="ignore"):
        pr = np.where(outdeg > 0, np.float32(1) / np.maximum(od, 1), np.float32(teleport)).astype(np.float32)
        for _ in range(sweeps):
            for v in range(len(outdeg)):
                x = pr[col[rp[v]:rp[v + 1]]]
                s = np.add.accumulate(x, dtype=np.float32)[-1] if x.size else np.float32(0)
                if x.size:  # the running sum starts at 0: 0 + x
                    s = np.add.accumulate(np.concatenate([np.zeros(1, np.float32), x]), dtype=np.float32)[-1]
                t = teleport + damping * float(s)
                pr[v] = np.float32(t / float(outdeg[v])) if outdeg[v] else np.float32(t)
        return np.where(outdeg > 0, pr * od, pr).astype(np.float32)


@pytest.mark.parametrize("teleport,damping", [
    (0.15, 0.85), (1.0, 1.0), (0.0, 0.5), (0.0, 0.0), (-0.3, 0.85), (-2.0, -0.9), (1e-39, 1e-7), (3e37, 0.9),
    (float("inf"), 0.5), (float("nan"), 0.5)])
def test_sequential_sums(teleport, damping):
    import gcgpu
    s, d = rows_graph(1)
    with gcgpu.Graph.from_edges(s, d, num_vertices=N, dedup=True, out_csr=False) as g:
        rp, col = g.csr()
        outdeg = g.degrees()[:, 1]
        got, st = g.pagerank(mode=gcgpu.PR_GS_EXACT, max_sweeps=2, teleport=teleport, damping=damping)
        assert st.levels > 1
        ref = restated(rp.astype(np.int64), col, outdeg, 2, teleport, damping)
        assert np.array_equal(got.view(np.uint32)[~np.isnan(ref)], ref.view(np.uint32)[~np.isnan(ref)])
        assert np.array_equal(np.isnan(got), np.isnan(ref))
