"""Products on invalid window ids (a caller's input of the strict-balance calls): the error word
says that an index was skipped and no wait ran out, and nothing outside C and the workspace is
written, whatever the ids are."""
import ctypes as C

import numpy as np
import pytest

from dtc_b200 import gen

pytestmark = pytest.mark.gpu


def _bad(rowid, nwin, kind):
    """`kind` of invalid ids from valid ones (sorted, 0 .. nwin - 1)."""
    rng = np.random.default_rng(3)
    r = rowid.copy()
    T = len(r)
    if kind == "first_negative":
        r[:2] = -50
    elif kind == "all_negative":
        r[:] = -1
    elif kind == "last_too_large":
        r[-3:] = nwin + 1000
    elif kind == "all_too_large":
        r[:] = nwin
    elif kind == "descending":
        r = r[::-1].copy()
    elif kind == "swapped":
        i = rng.choice(T, 40)
        r[i] = r[rng.permutation(i)]
    else:
        r = rng.integers(-3, nwin + 3, T).astype(np.int32)
    return r


@pytest.mark.parametrize("noalloc", [False, True])
@pytest.mark.parametrize("N", [32, 41, 128, 256])
@pytest.mark.parametrize("kind", ["first_negative", "all_negative", "last_too_large",
                                  "all_too_large", "descending", "swapped", "random"])
def test_product_stays_inside_its_arrays(cuda, kind, N, noalloc):
    import torch
    from dtc_b200 import _lib, metcf
    A = gen.zipf(6000, seed=5)
    m = metcf.convert(A.rowptr, A.col, A.M, values=A.val)
    rowid = torch.from_numpy(_bad(m.TCblockRowid.cpu().numpy(), m.nwin, kind)).cuda()
    B = torch.randn(A.M, N, device="cuda")
    pad = 32 * N  # two windows of C on each side
    buf = torch.full((A.M * N + 2 * pad,), 7.0, device="cuda")
    out = buf[pad:pad + A.M * N]
    wsb = metcf.spmm_balance_workspace_bytes(m, N)
    ws = torch.full((wsb + 2 * 65536,), 0x5a, dtype=torch.uint8, device="cuda")
    p = lambda t, off=0: C.c_void_p(t.data_ptr() + off)  # noqa: E731
    args = [p(rowid), p(m.TCblocktileId), p(m.TCblockoffset), p(m.SparseAToX), p(m.TCvalues), m.M,
            m.T, p(B), N, p(out)]
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    metcf.device_status(clear=True)
    L = _lib.lib()
    if noalloc:
        rc = L.dtc_spmm_balance_noalloc(*args, stream)
    else:
        rc = L.dtc_spmm_balance(*args, p(ws, 65536), wsb, stream)
    assert rc == 0
    assert metcf.device_status(clear=True) == 2
    assert (buf[:pad] == 7).all() and (buf[pad + A.M * N:] == 7).all()
    assert (ws[:65536] == 0x5a).all() and (ws[65536 + wsb:] == 0x5a).all()
