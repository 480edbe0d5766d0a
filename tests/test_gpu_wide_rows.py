"""GPU: index lists longer than the common forward kernel's tables (row-major K/V) on the tcgen05 kernel, against the scalar
kernel on the same inputs and mask: just past the common limit, at the variant's limit, both head sizes and element types, rows
that are nearly dense, empty, or hold one narrow block."""
import pytest
import torch

import cases as C

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("D,nk,bn,dt", [(128, 1468, 32, torch.bfloat16), (64, 1468, 32, torch.float16), (128, 4091, 32, torch.bfloat16),
                                        (64, 4091, 32, torch.bfloat16), (128, 2363, 32, torch.float16), (128, 1500, 64, torch.bfloat16)])
def test_wide_rows_equal_the_scalar_kernel(D, nk, bn, dt):
    from psa_b200 import ops
    S, Sq, H = nk * bn - 3, 128 * 5 + 7, 1
    k, v = (C.randn(800 + i, (1, H, S, D), dt).to(DEV) for i in range(2))
    q = C.randn(803, (1, H, Sq, D), dt).to(DEV)
    mq = -(-Sq // 128)
    g = torch.Generator().manual_seed(nk)
    mask = torch.zeros((1, H, mq, nk + 5), dtype=torch.int32)
    counts = [(nk // 2, nk // 4, nk // 8, nk - nk // 2 - nk // 4 - nk // 8), (40, 30, 20, 10), (0, 0, 0, 1), (0, 0, 0, 0), (1, 0, 2, 0), (0, nk, 0, 0)]
    for r in range(mq):
        blocks = torch.randperm(nk, generator=g).to(torch.int32)
        at, row = 0, []
        for c in counts[r]:
            row += blocks[at:at + c].tolist() + [-1]
            at += c
        mask[0, 0, r, :len(row)] = torch.tensor(row, dtype=torch.int32)
    mask = mask.to(DEV)
    assert mask.shape[-1] > 1472 and mask.shape[-1] <= 4096
    tc = ops.psa_forward(q, k, v, mask, 128, bn, 32)
    assert int(tc._psa_status.item()) == 0
    sc = ops.psa_forward(q, k, v, mask, 128, bn, 32, impl=ops.IMPL_SCALAR)
    tc, sc = tc.float(), sc.float()
    assert torch.equal(torch.isnan(tc), torch.isnan(sc))
    tc, sc = tc.nan_to_num(), sc.nan_to_num()
    # probabilities and results rounded to 8 (bf16) or 11 bits by both; a probability relative to another reference rounds anew
    assert float((tc - sc).abs().max()) <= 2e-2 and float((tc - sc).norm()) <= 1e-2 * float(sc.norm())
