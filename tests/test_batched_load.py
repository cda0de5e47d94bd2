"""BatchedSpMM.load: whole operands in one launch give what operand-by-operand copies give,
and operands that need those (shorter, other types, strided, from the host) still take them."""
import numpy as np
import pytest

from dtc_b200 import batched, gen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["whole", "fewer", "shorter", "double", "strided", "host", "grad"])
def test_load_forms(cuda, form):
    import torch
    mats = [gen.uniform(r, mean=4.0, seed=r) for r in (1, 15, 16, 17, 300, 4096)]
    N = 8
    plan = batched.BatchedSpMM(mats, N)
    plan.load([torch.full((m.M, N), 7.0, device="cuda") for m in mats])
    Bs = [torch.from_numpy(gen.normal(m.M, N, seed=i)).cuda() for i, m in enumerate(mats)]
    want = plan.B.clone()
    if form == "fewer":
        Bs = Bs[:2]
    elif form == "shorter":
        Bs[4] = Bs[4][:100]
    elif form == "double":
        Bs[3] = Bs[3].double()
    elif form == "strided":
        Bs[5] = Bs[5].t().contiguous().t()
    elif form == "host":
        Bs = [b.cpu() for b in Bs]
    elif form == "grad":
        Bs = [b.requires_grad_() for b in Bs]
    for o, b in zip(plan.layout.offsets, Bs):
        want[int(o):int(o) + b.shape[0]] = b.detach().to("cuda", torch.float32)
    with torch.no_grad():
        plan.load(b for b in Bs)
    np.testing.assert_array_equal(plan.B.detach().cpu().numpy(), want.cpu().numpy())


def test_load_fills_the_operand_that_the_plan_has(cuda):
    """A caller may put another tensor in place of the stacked operand."""
    import torch
    from dtc_b200 import gen
    from dtc_b200.batched import BatchedSpMM
    mats = [gen.uniform(n, mean=4.0, seed=n) for n in (33, 70, 16)]
    plan = BatchedSpMM(mats, 32)
    Bs = [torch.randn(m.M, 32, device="cuda") for m in mats]
    plan.load(Bs)
    old, want = plan.B, plan.B.clone()
    C = plan.run().clone()
    plan.B = torch.zeros_like(old)
    old.fill_(float("nan"))
    plan.load(Bs)
    assert torch.equal(plan.B, want) and torch.equal(plan.run(), C)
