"""The radix sort's way out when the counts of the tiles before do not come: every tile counts
again what it would have been told, over single tiles, whole groups of sixteen, and back to the
start. The graph is the one that the counts give."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "..", "graphchi-cpp_b200"))

pytestmark = pytest.mark.gpu

TILE = 256 * 22


def build(s, d, n, flags):
    import ctypes as C
    import gcgpu
    h = C.c_void_p()
    gcgpu.check(gcgpu._graph_from_edges(gcgpu.ptr(s), gcgpu.ptr(d), len(s), n, flags, 1, C.byref(h)))
    with gcgpu.Graph(h) as g:
        return g.csr() + (g.degrees(),)


@pytest.mark.parametrize("out_csr", [True, False])
@pytest.mark.parametrize("n", [200, 3000, 70_000])  # passes of one, and of several digits
@pytest.mark.parametrize("m", [1, TILE - 1, TILE, TILE + 1, 3 * TILE + 17, 16 * TILE, 16 * TILE + 1, 41 * TILE + 100])
def test_counted_again(m, n, out_csr):
    import gcgpu
    rng = np.random.default_rng(m + n)
    s, d = (rng.integers(0, n, m).astype(np.uint32) for _ in range(2))
    flags = gcgpu.BUILD_DEDUP | (0 if out_csr else gcgpu.BUILD_NO_OUT_CSR)
    rp, col, deg = build(s, d, n, flags | gcgpu.BUILD_TEST_RECOUNT)
    keys = np.unique(d[s != d].astype(np.int64) * n + s[s != d])
    assert np.array_equal(rp, np.concatenate([[0], np.cumsum(np.bincount(keys // n, minlength=n))]))
    assert np.array_equal(col, (keys % n).astype(np.uint32))
    assert np.array_equal(deg[:, 1], np.bincount(keys % n, minlength=n))
    for x, y in zip((rp, col, deg), build(s, d, n, flags)):
        assert np.array_equal(x, y)


def test_one_digit_over_all_tiles():
    import gcgpu
    m = 35 * TILE
    s, d = np.full(m, 7, np.uint32), np.arange(m, dtype=np.uint32) % np.uint32(5)
    rp, col, deg = build(s, d, 8, gcgpu.BUILD_NO_OUT_CSR | gcgpu.BUILD_TEST_RECOUNT)
    assert np.array_equal(np.diff(rp), np.bincount(d, minlength=8)) and (col == 7).all() and deg[7, 1] == m
