"""Products without a workspace: clusters of CTAs that add up the pieces of cut windows. Windows of
many chunks (several rounds of a cluster), several such windows in a row, at the start and at the
end, empty windows around them: the same bits as with a workspace, with and without the epilogue,
and within the form's bound (those of tests/test_spmm_shapes.py)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = {"tf32": 2.0 ** -9, "bf16x2x3": 2.0 ** -14, "split24x4": 2.0 ** -14, "bf16": 2.0 ** -8,
       "fp8": None}


@pytest.fixture(scope="module")
def hubs():
    """Windows 0-2, 90 and the last but one of all columns, every 7th window empty."""
    M = 6011
    rng = np.random.default_rng(11)
    rows = []
    for i in range(M):
        w = i // 32
        if w in (0, 1, 2, 90) or w == M // 32 - 1:
            n = M // 4
        elif w % 7 == 3 or w == M // 32:
            n = 0
        else:
            n = int(rng.integers(0, 25))
        rows.append(np.sort(rng.choice(M, size=n, replace=False)))
    rp = np.zeros(M + 1, np.int32)
    rp[1:] = np.cumsum([len(r) for r in rows])
    col = np.concatenate(rows).astype(np.int32)
    return rp, col, rng.uniform(-1, 1, col.size).astype(np.float32), M


@pytest.mark.parametrize("H,W", [(16, 8), (32, 8), (16, 16)])
@pytest.mark.parametrize("form,N", [("tf32", 20), ("tf32", 64), ("tf32", 128), ("tf32", 200),
                                    ("tf32", 516), ("bf16x2x3", 48), ("bf16x2x3", 128),
                                    ("bf16x2x3", 304), ("split24x4", 80), ("split24x4", 272),
                                    ("bf16", 128), ("bf16", 512), ("fp8", 144)])
def test_same_bits_as_with_a_workspace(cuda, hubs, form, N, H, W):
    import torch
    from dtc_b200 import metcf, tune
    rp, col, val, M = hubs
    m = metcf.convert(rp, col, M, H=H, W=W, values=val)
    B = np.random.default_rng(N).standard_normal((M, N)).astype(np.float32)
    Bd, bias = torch.from_numpy(B).cuda(), torch.randn(N, device="cuda")
    fmt, prec = tune.FORMS[form][:2]
    planes = [Bd] if form == "tf32" else metcf.pack_b(Bd, fmt)
    none = torch.empty(1, dtype=torch.uint8, device="cuda")

    def run(ws, **kw):
        out = torch.full((M, N), float("nan"), device="cuda")
        return metcf.spmm_fused(m, planes, fmt, N, prec, out=out, workspace=ws, **kw)
    one = run(none)
    assert torch.equal(one, run(None))
    assert torch.equal(run(none, bias=bias, relu=True), run(None, bias=bias, relu=True))
    assert metcf.device_status(clear=True) == 0
    if TOL[form]:
        err = np.abs(one.cpu().numpy().astype(np.float64) - O.spmm_f64(rp, col, val, M, B))
        assert (err <= TOL[form] * O.spmm_absbound_f64(rp, col, val, M, B) + 1e-6).all(), err.max()


@pytest.mark.parametrize("N", [1, 33, 129, 258])
def test_odd_widths_without_a_workspace(cuda, hubs, N):
    import torch
    from dtc_b200 import metcf
    from dtc_b200._lib import call
    from dtc_b200.metcf import _ptr, _stream
    rp, col, val, M = hubs
    m = metcf.convert(rp, col, M, values=val)
    B = torch.randn(M, N, device="cuda")
    out = torch.full((M, N), float("nan"), device="cuda")
    call("dtc_spmm", _ptr(m.RowWindowOffset), _ptr(m.TCblocktileId), _ptr(m.TCblockoffset),
         _ptr(m.SparseAToX), _ptr(m.TCvalues), m.M, m.nwin, m.T, _ptr(B), N, _ptr(out), _stream())
    assert torch.equal(out, metcf.spmm(m, B))
    # the strict-balance call without a workspace has two tiles per SM (fewer chunks)
    two = torch.full((M, N), float("nan"), device="cuda")
    call("dtc_spmm_balance_noalloc", _ptr(m.TCblockRowid), _ptr(m.TCblocktileId),
         _ptr(m.TCblockoffset), _ptr(m.SparseAToX), _ptr(m.TCvalues), m.M, m.T, _ptr(B), N,
         _ptr(two), _stream())
    Bh = B.cpu().numpy()
    bound = O.spmm_absbound_f64(rp, col, val, M, Bh)
    ref = O.spmm_f64(rp, col, val, M, Bh)
    for C in (out, two):
        assert (np.abs(C.cpu().numpy() - ref) <= 2.0 ** -9 * bound + 1e-6).all()
    assert metcf.device_status(clear=True) == 0
