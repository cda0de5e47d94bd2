"""Products of a matrix without edges: C = act(bias) through every entry point that takes one, and
zeros through the others."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("relu", [False, True])
@pytest.mark.parametrize("M,N", [(1, 16), (50, 32), (4099, 128), (70001, 48)])
def test_bias_of_an_edgeless_matrix(cuda, M, N, relu):
    import DTCSpMM
    import torch
    from dtc_b200 import B_F32, PREC_TF32, metcf, tune
    m = metcf.convert(torch.zeros(M + 1, dtype=torch.int32), torch.zeros(0, dtype=torch.int32), M)
    assert m.T == 0
    X, W, b = (torch.randn(*s, device="cuda") for s in ((M, 24), (24, N), (N,)))
    B = torch.randn(M, N, device="cuda")
    want = (torch.relu(b) if relu else b).expand(M, N)
    assert torch.equal(metcf.gcn_layer(m, X, W, bias=b, relu=relu), want)
    for form in ("tf32", "bf16x2x3"):
        fmt, prec = tune.FORMS[form][:2]
        planes = [B] if form == "tf32" else metcf.pack_b(B, fmt)
        out = torch.full((M, N), float("nan"), device="cuda")
        assert torch.equal(metcf.spmm_fused(m, planes, fmt, N, prec, bias=b, relu=relu, out=out), want)
    arrays = (m.RowWindowOffset, m.TCblocktileId, m.TCblockoffset, m.SparseAToX, M, 0)
    assert torch.equal(DTCSpMM.DTCSpMM_gcn(B, *arrays, bias=b, relu=relu)[0], want)
    for C in (metcf.spmm_fused(m, [B], B_F32, N, PREC_TF32, relu=relu), metcf.spmm(m, B),
              metcf.spmm_balance(m, B)):
        assert torch.equal(C, torch.zeros_like(B))
