"""Relabelling at the edges of its tiles of 2048 edges: rows that start or end there, long
runs of empty rows, hub rows over several tiles, with and without equal pairs (which take a
second, merging pass) and values. Bit-exact with the oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _csr(M, K, nnz, equal, seed):
    rng = np.random.default_rng(seed)
    r = np.sort(np.where(rng.random(nnz) < 0.5, M // 3, rng.integers(0, M, nnz)))
    c = rng.integers(0, K, nnz)
    if not equal:  # distinct pairs, columns of a row in any order
        _, first = np.unique(r * K + c, return_index=True)
        free = np.setdiff1d(np.arange((M // 3) * K, (M // 3) * K + K), r * K + c)
        keep = np.zeros(nnz, bool)
        keep[first] = True
        fill = rng.choice(free, nnz - first.size, replace=False)
        r = np.concatenate([r[keep], fill // K])
        c = np.concatenate([c[keep], fill % K])
        o = np.argsort(r, kind="stable")
        r, c = r[o], c[o]
    rowptr = np.searchsorted(r, np.arange(M + 1)).astype(np.int32)
    return rowptr, r.astype(np.int32), c.astype(np.int32), rng.standard_normal(nnz).astype(np.float32)


@pytest.mark.parametrize("equal", [False, True])
@pytest.mark.parametrize("with_values", [False, True])
@pytest.mark.parametrize("M,nnz", [(1, 1), (7, 2047), (5000, 2048), (5000, 2049), (300000, 9000)])
def test_tiles(cuda, M, nnz, with_values, equal):
    import torch
    from dtc_b200 import dataset, metcf
    K = max(M, 20000)
    rowptr, r, c, val = _csr(M, K, nnz, equal, seed=nnz)
    v = val if with_values else None
    g = lambda x: None if x is None else torch.from_numpy(x).cuda()
    same = lambda got, exp: [np.testing.assert_array_equal(a.cpu().numpy(), b)
                             for a, b in zip(got, exp)]
    same(metcf.transpose_csr(g(rowptr), g(c), g(v), K), O.transpose_csr(rowptr, c, v, K))
    mix = np.random.default_rng(1).permutation(nnz)
    vm = None if v is None else v[mix]
    same(dataset.coo_to_csr(r[mix], c[mix], M, K, val=vm), O._coo_to_csr(r[mix], c[mix], vm, M, K))
    square = np.concatenate([rowptr, np.full(K - M, nnz, np.int32)])
    perm = np.random.default_rng(2).permutation(K).astype(np.int32)
    same(metcf.permute_csr(g(square), g(c), g(v), g(perm)), O.permute_csr(square, c, v, perm))
