"""The sharder's sort and its last pass at the edges of their tiles: 5632 keys per
sort tile, 16 tiles per group of the look-back, 512 keys per warp of the finish.
Id ranges of 16 and 22 bits count the out-degrees between two passes, 17 bits
(odd pass count) from the columns; a source array that starts 4 bytes past a
16-byte boundary takes the scalar edge scan. Whole numbers: compared exactly with
numpy's sort."""
import numpy as np
import pytest

import gcgpu
import oracle as O

pytestmark = pytest.mark.gpu

TILE, GROUP, SEG = 5632, 16 * 5632, 512


@pytest.mark.parametrize("bits", [3, 16, 17, 22])
@pytest.mark.parametrize("m", [1, SEG - 1, SEG + 1, TILE - 1, TILE, TILE + 1, GROUP - 1, GROUP + 1,
                               3 * GROUP + 2 * TILE + 7])
@pytest.mark.parametrize("dedup", [True, False])
def test_sorted_edges_equal_numpy(bits, m, dedup):
    import torch
    rng = np.random.default_rng(m * 64 + bits)
    n = 1 << bits
    s, d = rng.integers(0, n, (2, m), dtype=np.uint32)
    hub = rng.random(m) < 0.3
    d[hub] = n - 1  # a row that spans tiles; with s = n - 1 also the ids of the self-loop sentinel
    s[rng.random(m) < 0.1] = n - 1
    rep = rng.integers(0, m, m // 4)
    s[rep], d[rep] = s[rep[::-1]], d[rep[::-1]]
    ts = torch.from_numpy(np.concatenate([[0], s]).astype(np.int64)).to(torch.int32).cuda()[1:]
    td = torch.from_numpy(d.astype(np.int64)).to(torch.int32).cuda()
    keep = s != d
    k = (d[keep].astype(np.uint64) << np.uint64(32)) | s[keep]
    k = np.unique(k) if dedup else np.sort(k)
    row, col = (k >> np.uint64(32)).astype(np.int64), (k & np.uint64(0xFFFFFFFF)).astype(np.uint32)
    with gcgpu.Graph.from_edges(ts, td, num_vertices=n, dedup=dedup, nshards=5, out_csr=False) as g:
        assert g.num_edges == k.shape[0]
        rp, c = g.csr(gcgpu.CSR_IN)
        assert np.array_equal(c, col)
        assert np.array_equal(rp, np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]))
        deg = g.degrees()
        assert np.array_equal(deg[:, 0], np.bincount(row, minlength=n))
        assert np.array_equal(deg[:, 1], np.bincount(col.astype(np.int64), minlength=n))


def test_reference_intervals_of_uneven_rows():
    """Cuts that fall exactly on a row's start, inside long rows and among empty rows."""
    rng = np.random.default_rng(5)
    d = np.repeat(rng.permutation(70000)[:3000], rng.integers(1, 400, 3000)).astype(np.uint32)
    s = rng.integers(70000, 80000, d.shape[0], dtype=np.uint32)
    o = O.OracleGraph(s, d)
    for p in (2, 7, 64, 5000):
        with gcgpu.Graph.from_edges(s, d, dedup=True, nshards=p, out_csr=False) as g:
            assert np.array_equal(g.intervals(), o.intervals(p)), p
