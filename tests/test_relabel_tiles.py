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


@pytest.mark.parametrize("fault", ["perm", "rowptr", "col", "row", "col_coo"])
def test_outputs_of_a_refused_call_stay_as_they_are(cuda, fault):
    import ctypes as C
    import torch
    from dtc_b200 import _lib
    from dtc_b200.metcf import _ptr, _stream
    M, nnz = 30000, 20000
    rowptr, r, c, val = _csr(M, M, nnz, False, seed=4)
    perm = np.arange(M, dtype=np.int32)
    if fault == "perm":
        perm[5] = perm[6]
    elif fault == "rowptr":
        rowptr[M // 2] = nnz + 1
    elif fault == "row":
        r[77] = M
    else:
        c[nnz - 1] = -1
    g = lambda x: torch.from_numpy(x).cuda()
    L = _lib.lib()
    b = C.c_size_t()
    assert L.dtc_relabel_workspace_bytes(M, M, nnz, C.byref(b)) == 0
    ws = torch.empty(b.value, dtype=torch.uint8, device="cuda")
    rp = torch.full((M + 1,), -5, dtype=torch.int32, device="cuda")
    co = torch.full((nnz,), -5, dtype=torch.int32, device="cuda")
    vo = torch.full((nnz,), -5.0, device="cuda")
    n = C.c_int64(-5)
    inputs = [g(rowptr), g(c), g(val), g(perm), g(r)]
    p = [_ptr(t) for t in inputs]
    outs = [_ptr(rp), _ptr(co), _ptr(vo), C.byref(n), _ptr(ws), b.value, _stream()]
    calls = {"perm": lambda: L.dtc_permute_csr(*p[:3], M, nnz, p[3], *outs),
             "csr": lambda: L.dtc_transpose_csr(*p[:3], M, M, nnz, *outs),
             "coo": lambda: L.dtc_coo_to_csr(p[4], p[1], p[2], M, M, nnz, *outs)}
    for name in {"perm": ["perm"], "rowptr": ["perm", "csr"], "col": ["perm", "csr"], "row": ["coo"],
                 "col_coo": ["coo"]}[fault]:
        assert calls[name]() == 1
        assert n.value == -5
        for t in (rp, co, vo):
            assert (t == -5).all()


@pytest.mark.parametrize("equal", [False, True])
@pytest.mark.parametrize("first,gap,last", [(0, 33, 0), (5, 32, 1), (1, 5000, 300), (70000, 1, 70000)])
def test_long_runs_of_empty_rows(cuda, first, gap, last, equal):
    import torch
    from dtc_b200 import dataset, metcf
    # 3000 entries in two groups of rows, with runs of empty rows before, between and after them
    rng = np.random.default_rng(gap)
    rows = 600 + first + gap + last
    r = first + rng.integers(0, 300, 3000)
    r[1500:] += 300 + gap
    c = rng.integers(0, 40 if equal else 1 << 20, 3000)
    if not equal:
        c = (c // 3000 * 3000 + np.arange(3000)).astype(np.int64)
    val = rng.standard_normal(3000).astype(np.float32)
    got = dataset.coo_to_csr(r.astype(np.int32), c.astype(np.int32), rows, 1 << 21, val=val)
    exp = O._coo_to_csr(r.astype(np.int32), c.astype(np.int32), val, rows, 1 << 21)
    for a, b in zip(got, exp):
        np.testing.assert_array_equal(a.cpu().numpy(), b)
    # the same rows as the columns of a matrix to transpose
    o = np.argsort(c, kind="stable")
    rp = np.searchsorted(c[o], np.arange((1 << 21) + 1)).astype(np.int32)
    g = lambda x: torch.from_numpy(x).cuda()
    got = metcf.transpose_csr(g(rp), g(r[o].astype(np.int32)), g(val[o]), rows)
    exp = O.transpose_csr(rp, r[o].astype(np.int32), val[o], rows)
    for a, b in zip(got, exp):
        np.testing.assert_array_equal(a.cpu().numpy(), b)
