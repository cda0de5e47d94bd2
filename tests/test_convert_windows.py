"""ME-TCF conversion at the edges of its window classes (edges of a window sorted by one
warp, by one CTA, ranked by a bitmap; placed by one warp, in units, row by row): bit-exact
with the oracle, integers and merged values alike."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

COUNTS = [0, 1, 31, 33, 128, 129, 256, 257, 512, 513, 1024, 1025, 2048, 2049, 16384, 16385, 40000]


def _matrix(M, H, order, seed=0):
    """Windows of COUNTS edges spread over the rows, the last one on the last window."""
    rng = np.random.default_rng(seed)
    nwin = (M + H - 1) // H
    deg = np.zeros(M, np.int64)
    rows = {}
    for i, n in enumerate(COUNTS):
        w = (nwin - 1) * i // (len(COUNTS) - 1)
        r0, r1 = w * H, min(w * H + H, M)
        share = rng.multinomial(n, rng.dirichlet(np.ones(r1 - r0)))
        for r, d in zip(range(r0, r1), share):
            if order == "mixed" and r % 3:  # repeated and unsorted columns
                c = rng.integers(0, max(1, M // 7), d)
            else:
                c = np.sort(rng.choice(M, d, replace=False)) if d else np.empty(0, np.int64)
            rows[r], deg[r] = c, d
    rowptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    col = np.concatenate([rows[r] for r in sorted(rows)]).astype(np.int32)
    return rowptr, col, rng.random(col.size).astype(np.float32)


@pytest.mark.parametrize("order", ["ascending", "mixed"])
@pytest.mark.parametrize("M,H,W", [(60001, 16, 8), (60001, 32, 8), (60001, 16, 16), (60001, 1, 256),
                                   (60001, 5, 7), (60001, 64, 4), (60001, 256, 1),
                                   (2 ** 21 + 5, 16, 8)])
def test_window_classes(cuda, M, H, W, order):
    from dtc_b200 import metcf
    rowptr, col, val = _matrix(M, H, order)
    got = metcf.convert(rowptr, col, M, H=H, W=W, values=val)
    exp = O.metcf(rowptr, col, M, H=H, W=W, values=val)
    assert got.T == exp["T"]
    for k in ("RowWindowOffset", "TCblockRowid", "TCblocktileId", "TCblockoffset", "SparseAToX",
              "blockPartition", "edgeToColumn", "edgeToRow", "TCvalues"):
        np.testing.assert_array_equal(getattr(got, k).cpu().numpy(), exp[k], err_msg=k)


@pytest.mark.parametrize("order", ["ascending", "mixed"])
@pytest.mark.parametrize("M,H,W", [(70001, 1, 8), (70001, 2, 8), (70001, 16, 8), (70001, 16, 16),
                                   (70001, 7, 5), (70001, 32, 8), (300001, 256, 1),
                                   (2 ** 22 + 3, 3, 8), (2 ** 19 + 7, 1, 256)])
def test_few_edges_per_window(cuda, M, H, W, order):
    """At most 16 edges per window on average: windows of up to 16 edges by one lane, the others
    as in other matrices; the last matrix has windows enough for the two-level scan."""
    from dtc_b200 import metcf
    rng = np.random.default_rng(M + H)
    nwin = (M + H - 1) // H
    n = rng.integers(0, 18, nwin)
    n[:4] = 16, 17, 1, 0
    n[rng.choice(nwin, 3, replace=False)] = 300
    n[-1] = 15
    if nwin > 1200:
        n[nwin // 2], n[nwin // 3] = 1100, 2500
    n = np.minimum(n, 8 * M // nwin + 9)
    w = np.repeat(np.arange(nwin), n)
    row = np.minimum(w * H + rng.integers(0, H, w.size), M - 1)
    few = rng.random(w.size) < 0.3
    col = np.where(few, rng.integers(0, 9, w.size), rng.integers(0, M, w.size))
    o = np.lexsort((col if order == "ascending" else rng.random(w.size), row))
    row, col = row[o], col[o]
    if order == "ascending":  # distinct
        keep = np.r_[True, (row[1:] != row[:-1]) | (col[1:] != col[:-1])]
        row, col = row[keep], col[keep]
    rowptr = np.searchsorted(row, np.arange(M + 1)).astype(np.int32)
    assert col.size <= 16 * nwin
    col, val = col.astype(np.int32), rng.random(col.size).astype(np.float32)
    got = metcf.convert(rowptr, col, M, H=H, W=W, values=val)
    exp = O.metcf(rowptr, col, M, H=H, W=W, values=val)
    assert got.T == exp["T"]
    for k in ("RowWindowOffset", "TCblockRowid", "TCblocktileId", "TCblockoffset", "SparseAToX",
              "blockPartition", "edgeToColumn", "edgeToRow", "TCvalues"):
        np.testing.assert_array_equal(getattr(got, k).cpu().numpy(), exp[k], err_msg=k)


@pytest.mark.parametrize("H,W", [(16, 8), (32, 8), (16, 16), (64, 4), (3, 64)])
@pytest.mark.parametrize("n", [300, 1000, 9000, 40000, 200000])
def test_unsorted_windows_with_hot_columns(cuda, n, H, W):
    """Edges in any order, a few columns that most of them repeat (blocks of thousands of edges,
    merged values) and many more that occur once."""
    from dtc_b200 import metcf
    M = 50000
    rng = np.random.default_rng(n + H)
    row = np.repeat([M // 2 // H * H, M // 2 // H * H + H - 1, M - 1], [n // 2, n // 4, n // 4])
    col = np.where(rng.random(row.size) < 0.7, rng.integers(700, 703, row.size),
                   rng.integers(0, M, row.size))
    rowptr = np.searchsorted(row, np.arange(M + 1)).astype(np.int32)
    col, val = col.astype(np.int32), rng.standard_normal(col.size).astype(np.float32)
    got = metcf.convert(rowptr, col, M, H=H, W=W, values=val)
    exp = O.metcf(rowptr, col, M, H=H, W=W, values=val)
    assert got.T == exp["T"]
    for k in ("RowWindowOffset", "TCblockRowid", "TCblocktileId", "TCblockoffset", "SparseAToX",
              "blockPartition", "edgeToColumn", "edgeToRow", "TCvalues"):
        np.testing.assert_array_equal(getattr(got, k).cpu().numpy(), exp[k], err_msg=k)


@pytest.mark.parametrize("M", [2 ** 20 + 1, 2 ** 22 + 3, 2 ** 23 + 5])
@pytest.mark.parametrize("H", [1, 16, 64])
def test_large_windows_of_many_columns(cuda, M, H):
    """Matrices of more columns than one bitmap has bits: windows sorted by a CTA up to a size that
    grows with the columns, beyond it ranked by several bitmaps."""
    from dtc_b200 import metcf
    rng = np.random.default_rng(M + H)
    nwin = (M + H - 1) // H
    counts = [1024, 1025, 2047, 2048, 2049, 4096, 4097, 8192, 8193, 16384, 16385, 30000]
    row = np.concatenate([np.minimum((nwin - 1) * (i + 1) // len(counts) * H + rng.integers(0, H, n), M - 1)
                          for i, n in enumerate(counts)])
    col = rng.integers(0, M, row.size)
    col[rng.random(row.size) < 0.1] = M - 1
    o = np.lexsort((col, row))
    row, col = row[o], col[o].astype(np.int32)
    rowptr = np.searchsorted(row, np.arange(M + 1)).astype(np.int32)
    val = rng.random(col.size).astype(np.float32)
    got = metcf.convert(rowptr, col, M, H=H, W=4, values=val)
    exp = O.metcf(rowptr, col, M, H=H, W=4, values=val)
    assert got.T == exp["T"]
    for k in ("RowWindowOffset", "TCblockRowid", "TCblocktileId", "TCblockoffset", "SparseAToX",
              "blockPartition", "edgeToColumn", "edgeToRow", "TCvalues"):
        np.testing.assert_array_equal(getattr(got, k).cpu().numpy(), exp[k], err_msg=k)
