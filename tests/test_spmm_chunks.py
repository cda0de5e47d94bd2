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
