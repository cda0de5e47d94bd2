"""Workspaces off the 16-byte boundary: the strict-balance calls take any 4-byte place (same bits)
and write nothing beyond the bytes that they ask for."""
import ctypes as C

import pytest

from dtc_b200 import gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("place", [4, 8, 12])
@pytest.mark.parametrize("form,N,H", [("tf32", 32, 16), ("tf32", 41, 16), ("tf32", 128, 16),
                                      ("tf32", 256, 16), ("tf32", 128, 32), ("bf16x2x3", 64, 16),
                                      ("bf16", 64, 32), ("split24x3", 128, 16), ("fp8", 80, 16)])
def test_required_bytes_at_any_place(cuda, form, N, H, place):
    import torch
    from dtc_b200 import _lib, metcf, tune
    from dtc_b200.metcf import _ptr, _stream
    A = gen.zipf(20000, seed=5)
    m = metcf.convert(A.rowptr, A.col, A.M, H=H, values=A.val)
    B = torch.randn(A.M, N, device="cuda")
    fmt, prec = tune.FORMS[form][:2]
    planes = [B] if form == "tf32" else metcf.pack_b(B, fmt)

    def run(call, need, at):
        ws = torch.full((need + 64,), 0xff, dtype=torch.uint8, device="cuda")
        out = torch.full((A.M, N), float("nan"), device="cuda")
        assert call(out, C.c_void_p(ws.data_ptr() + at), need) == 0, _lib.lib().dtc_last_error()
        assert (ws[:at] == 0xff).all() and (ws[at + need:] == 0xff).all()
        return out

    L = _lib.lib()
    arrays = [_ptr(m.TCblocktileId), _ptr(m.TCblockoffset), _ptr(m.SparseAToX), _ptr(m.TCvalues)]
    if form == "tf32" and H == 16:
        need = metcf.spmm_balance_workspace_bytes(m, N)

        def balance(out, ws, wsb):
            return L.dtc_spmm_balance(_ptr(m.TCblockRowid), *arrays, m.M, m.T, _ptr(B), N,
                                      _ptr(out), ws, wsb, _stream())
        assert torch.equal(run(balance, need, 0), run(balance, need, place))
    if N % 4:
        return
    need = metcf.spmm_ex_workspace_bytes(m, N, 1) - metcf.spmm_ex_workspace_bytes(m, N, 0)
    for more in (0, metcf.spmm_ex_workspace_bytes(m, N, 0)):

        def ex(out, ws, wsb):
            return L.dtc_spmm_ex(_ptr(m.RowWindowOffset), *arrays, m.M, m.nwin, m.T, m.H, m.W, fmt,
                                 _ptr(planes[0]), _ptr(planes[1]) if len(planes) > 1 else None, N,
                                 prec, _ptr(out), 1, 0, 0, ws, wsb, _stream())
        assert torch.equal(run(ex, need + more, 0), run(ex, need + more, place))
    assert metcf.device_status(clear=True) == 0
