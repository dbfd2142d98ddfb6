"""Batched PPR's segments, placed by counted lengths: rows around one and several segments of 256
in-edges, rows of more segments than are counted apart (4096), rows without in-edges, against
the sweeps in 64 bits."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "graphchi-cpp_b200"))

pytestmark = pytest.mark.gpu

MANY = 4096 * 256


@pytest.mark.parametrize("lengths,n", [
    ([1, 2, 255, 256, 257, 511, 512, 513, 767, 768, 769, 1, 3000, 256, 512], 5000),
    ([MANY - 1, 5, MANY, 300, MANY + 1, 0, MANY + 300, 256, MANY + 600], 1_100_000),
    ([0, 0, 0], 300), ([3], 40)])
def test_segments(lengths, n):
    import gcgpu
    rng = np.random.default_rng(1)
    rows = rng.choice(n, len(lengths), replace=False)
    src = np.concatenate([np.delete(np.arange(n), v)[:k] for v, k in zip(rows, lengths)] +
                         [rows, (rows + 1) % n]).astype(np.uint32)  # the rows feed some thin ones
    dst = np.concatenate([np.repeat(rows, lengths), (rows + 1) % n, (rows + 2) % n]).astype(np.uint32)
    sources = np.unique(np.concatenate([rows[:3], rng.choice(n, 4)])).astype(np.uint32)
    sweeps, tele, damp = 3, 0.15, 0.85
    with gcgpu.Graph.from_edges(src, dst, num_vertices=n, dedup=True, out_csr=False) as g:
        got, _ = g.ppr_batched(sources, max_sweeps=sweeps, teleport=tele, damping=damp)
        rp, col = g.csr()
        outdeg = g.degrees()[:, 1]
    row = np.repeat(np.arange(n), np.diff(rp.astype(np.int64)))
    share = np.where(outdeg > 0, 1.0 / np.maximum(outdeg, 1), 0.0)
    for j, s in enumerate(sources):
        r = np.zeros(n)
        r[s] = 1.0
        for _ in range(sweeps):
            r = damp * np.bincount(row, weights=(r * share)[col], minlength=n)
            r[s] += tele
        assert np.abs(got[:, j] - r).sum() <= 1e-6 * max(r.sum(), 1e-30), s
