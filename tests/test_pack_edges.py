"""Storage forms of B packed eight elements at a time: remainders, and buffers off the
16-byte boundary (an element per thread). Bit-exact with the oracle."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (4, 8, 16)])
@pytest.mark.parametrize("rows,N", [(1, 1), (1, 7), (3, 3), (2, 4), (17, 41), (500, 128)])
def test_pack_edges(cuda, rows, N, off):
    import torch
    from dtc_b200 import B_BF16, B_BF16X2, B_FP8, B_SPLIT24, metcf
    B = np.random.default_rng(rows * N).standard_normal((rows, N)).astype(np.float32)
    B.flat[0] = np.inf
    n = rows * N
    Bd = torch.empty(n + 8, device="cuda")[off[0]:off[0] + n].view(rows, N)
    Bd.copy_(torch.from_numpy(B))
    F = np.where(np.isfinite(B), B, np.float32(0)).astype(np.float32)
    for fmt, first, second, exp in ((B_SPLIT24, 2, 1, O.pack_split24(B)), (B_BF16, 2, 0, (O.pack_bf16(B),)),
                                    (B_BF16X2, 2, 2, O.pack_bf16x2(B)), (B_FP8, 1, 4, O.pack_fp8(F))):
        if fmt == B_FP8:
            Bd.copy_(torch.from_numpy(F))
        sizes = [s for s in (first, second) if s]
        raw = [torch.full((s * (n + 32),), 7, dtype=torch.uint8, device="cuda") for s in sizes]
        at = [s * o for s, o in zip(sizes, off[1:])]
        planes = [r[o:o + e.nbytes] for r, o, e in zip(raw, at, exp)]
        metcf.pack_b_into(Bd, fmt, planes)
        for r, o, e in zip(raw, at, exp):
            got = r.cpu().numpy()
            np.testing.assert_array_equal(got[o:o + e.nbytes].view(e.dtype).reshape(e.shape), e)
            assert (got[:o] == 7).all() and (got[o + e.nbytes:] == 7).all()
