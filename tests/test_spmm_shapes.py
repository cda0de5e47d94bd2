"""GPU parity of the SpMM kernels at the edges of their tiles: feature slices of
32, 64 and 128 (and 256 per CTA), every block shape and B form, windows cut
between warps and between CTAs, and the same bits with and without slots in the
workspace.

Tolerances are those of the forms' other tests: |C - C64| <= tol * sum |a||b| +
1e-6 with tol = 2^-9 (TF32: A to 11 bits, B cut to 11), 2^-14 (BF16X2, SPLIT24:
16 significant bits of A and B, three or four products), 2^-8 (BF16, and FP8
against B as stored).
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = {"tf32": 2.0 ** -9, "bf16x2x3": 2.0 ** -14, "split24x3": 2.0 ** -14,
       "split24x4": 2.0 ** -14, "bf16": 2.0 ** -8, "fp8": 2.0 ** -8}


def _skewed(M, seed=7):
    """Rows of 0-40 entries, a run of empty windows, and two hub windows of
    thousands of columns (windows of hundreds of blocks, cut between CTAs)."""
    rng = np.random.default_rng(seed)
    rows = []
    for i in range(M):
        if M // 3 <= i < M // 3 + 100:
            n = 0
        elif i // 16 in (6, M // 16 - 1):
            n = M // 3
        else:
            n = int(rng.integers(0, 41))
        rows.append(np.sort(rng.choice(M, size=min(n, M), replace=False)))
    rp = np.zeros(M + 1, np.int32)
    rp[1:] = np.cumsum([len(r) for r in rows])
    return rp, np.concatenate(rows).astype(np.int32), \
        rng.uniform(-1, 1, int(rp[-1])).astype(np.float32), M


@pytest.fixture(scope="module")
def skewed():
    return _skewed(4011)


def _run(mat, form, N, H, W, mode, slots=True):
    import torch
    from dtc_b200 import metcf, tune
    rp, col, val, M = mat
    m = metcf.convert(rp, col, M, H=H, W=W, values=val)
    B = np.random.default_rng(N).standard_normal((M, N)).astype(np.float32)
    Bd = torch.from_numpy(B).cuda()
    fmt, prec = tune.FORMS[form][:2]
    planes = [Bd] if form == "tf32" else metcf.pack_b(Bd, fmt)
    full = metcf.spmm_ex_workspace_bytes(m, N, mode)
    wsb = full if slots else full - metcf.spmm_ex_workspace_bytes(m, N, 0)
    ws = torch.full((max(wsb, 1),), 0xff, dtype=torch.uint8, device="cuda")
    out = torch.full((M, N), float("nan"), device="cuda")
    C = metcf.spmm_ex(m, planes, fmt, N, prec, mode=mode, workspace=ws, out=out)
    assert metcf.device_status(clear=True) == 0
    return C, B


def _check(C, mat, form, B):
    rp, col, val, M = mat
    if form == "fp8":
        q, s = O.pack_fp8(B)
        B = (O.e4m3_values(q) * s[:, None]).astype(np.float32)
    err = np.abs(C.cpu().numpy().astype(np.float64) - O.spmm_f64(rp, col, val, M, B))
    assert (err <= TOL[form] * O.spmm_absbound_f64(rp, col, val, M, B) + 1e-6).all(), err.max()


@pytest.mark.parametrize("H,W", [(16, 8), (32, 8), (16, 16)])
@pytest.mark.parametrize("form,N", [("tf32", n) for n in (4, 32, 36, 64, 68, 128, 132, 256, 260, 388)]
                         + [(f, n) for f in ("bf16x2x3", "bf16") for n in (16, 64, 80, 128, 144, 272)]
                         + [(f, n) for f in ("split24x3", "split24x4", "fp8") for n in (16, 80, 144)])
def test_slices(cuda, skewed, form, N, H, W):
    C, B = _run(skewed, form, N, H, W, mode=(N // 4) % 2)
    _check(C, skewed, form, B)


@pytest.mark.parametrize("N", [1, 3, 31, 33, 41, 65, 129, 257])
def test_odd_widths(cuda, skewed, N):
    import torch
    from dtc_b200 import metcf
    rp, col, val, M = skewed
    m = metcf.convert(rp, col, M, values=val)
    B = np.random.default_rng(N).standard_normal((M, N)).astype(np.float32)
    Bt = torch.from_numpy(B).cuda()
    C = metcf.spmm(m, Bt)
    _check(C, skewed, "tf32", B)
    _check(metcf.spmm_balance(m, Bt), skewed, "tf32", B)
    # B and C at any 4-byte place
    buf = torch.zeros(M * N + 1, device="cuda")
    view = buf[1:].view(M, N)
    view.copy_(Bt)
    assert torch.equal(metcf.spmm(m, view), C)


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("form,N,H", [("tf32", 32, 16), ("tf32", 128, 16), ("tf32", 128, 32),
                                      ("bf16x2x3", 64, 32), ("bf16x2x3", 256, 16),
                                      ("split24x3", 128, 16), ("fp8", 64, 16)])
def test_same_bits_without_slots(cuda, skewed, form, N, H, mode):
    import torch
    a, B = _run(skewed, form, N, H, 8, mode)
    b, _ = _run(skewed, form, N, H, 8, mode, slots=False)
    c, _ = _run(skewed, form, N, H, 8, mode)
    _check(a, skewed, form, B)
    assert torch.equal(a, b) and torch.equal(a, c)


@pytest.mark.parametrize("form,N", [("tf32", 64), ("tf32", 256), ("bf16x2x3", 128)])
def test_long_chunks(cuda, form, N):
    """Enough blocks for long chunks, whose last quarter is cut finer."""
    from dtc_b200 import gen
    A = gen.rmat(18, 16.0, seed=3)
    mat = (A.rowptr, A.col, A.val, A.M)
    C, B = _run(mat, form, N, 16, 8, 0)
    _check(C, mat, form, B)
