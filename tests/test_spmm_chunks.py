"""Products at block counts around which the chunk rule changes (no split of the last quarter,
one wave of chunks, chunks of fixed size): within the FP64 bound of TF32, and the same bits with
and without the workspace that holds the pieces of cut windows."""
import numpy as np
import pytest

from oracle import oracle as O
from dtc_b200 import gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [16, 132])
@pytest.mark.parametrize("rows", [4900, 5300, 24000, 28000])
def test_chunk_rule(cuda, rows, N):
    import torch
    from dtc_b200 import B_F32, PREC_TF32, metcf
    A = gen.uniform(rows, mean=47.0, seed=rows)
    m = metcf.convert(A.rowptr, A.col, A.M, values=A.val)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert (rows < 5000) == (m.T // (sms * 12) < 16) and (rows < 25000) == (m.T // (sms * 12) < 80)
    B = gen.normal(A.M, N, seed=1)
    Bd = torch.from_numpy(B).cuda()
    ws = torch.empty(metcf.spmm_ex_workspace_bytes(m, N), dtype=torch.uint8, device="cuda")
    one = metcf.spmm_ex(m, [Bd], B_F32, N, PREC_TF32, workspace=ws)
    two = metcf.spmm_ex(m, [Bd], B_F32, N, PREC_TF32, workspace=ws[:1])
    assert torch.equal(one, two)
    slot = 16 * N * 4  # (fewer slots: fewer chunks; less than one per SM: none)
    few = [metcf.spmm_ex(m, [Bd], B_F32, N, PREC_TF32, workspace=ws[:n * slot])
           for n in (sms - 1, sms, sms)]
    assert torch.equal(one, few[0]) and torch.equal(few[1], few[2])
    ref = O.spmm_f64(A.rowptr, A.col, A.val, A.M, B)
    bound = O.spmm_absbound_f64(A.rowptr, A.col, A.val, A.M, B)
    for C in (one, few[1]):
        assert (np.abs(C.cpu().numpy() - ref) <= 2.0 ** -9 * bound + 1e-6).all()


@pytest.mark.parametrize("form,N,H", [("tf32", 32, 16), ("tf32", 256, 16), ("tf32", 256, 32),
                                      ("bf16x2x3", 128, 32), ("bf16", 512, 16), ("split24x3", 144, 16)])
@pytest.mark.parametrize("rows,mean", [(9, 3.0), (40, 2.0), (100, 4.0), (700, 8.0), (1500, 6.0),
                                       (5000, 9.0), (7000, 40.0)])
def test_small_products(cuda, rows, mean, form, N, H):
    """Chunks of a few blocks, 128 of them, one wave of them."""
    import torch
    from dtc_b200 import metcf, tune
    A = gen.uniform(rows, mean=mean, seed=rows)
    m = metcf.convert(A.rowptr, A.col, A.M, H=H, values=A.val)
    B = gen.normal(A.M, N, seed=1)
    Bd = torch.from_numpy(B).cuda()
    fmt, prec = tune.FORMS[form][:2]
    planes = [Bd] if form == "tf32" else metcf.pack_b(Bd, fmt)
    C = metcf.spmm_ex(m, planes, fmt, N, prec)
    assert torch.equal(C, metcf.spmm_ex(m, planes, fmt, N, prec, workspace=torch.empty(
        1, dtype=torch.uint8, device="cuda")))
    tol = {"tf32": 2.0 ** -9, "bf16": 2.0 ** -8}.get(form, 2.0 ** -14)
    ref = O.spmm_f64(A.rowptr, A.col, A.val, A.M, B)
    bound = O.spmm_absbound_f64(A.rowptr, A.col, A.val, A.M, B)
    assert (np.abs(C.cpu().numpy() - ref) <= tol * bound + 1e-6).all()
    assert metcf.device_status(clear=True) == 0


def test_workspace_of_a_huge_matrix_is_bounded(cuda):
    """A slot per chunk, and at most 16384 chunks however many blocks there are."""
    import ctypes as C
    from dtc_b200 import _lib
    n = C.c_size_t()
    last = 0
    for blocks in (10 ** 5, 10 ** 6, 10 ** 7, 10 ** 8, 2 ** 31 - 1):
        assert _lib.lib().dtc_spmm_ex_workspace_bytes(1 << 24, blocks, 512, 32, 0, 0, C.byref(n)) == 0
        assert last <= n.value <= 16384 * 32 * 512 * 4
        last = n.value
