"""GPU: index lists of more than PSA_FWD_LIST_MAX entries (row-major K/V) on the tcgen05 kernel, against the scalar kernel on the same
inputs and mask: just past that limit, at PSA_FWD_LIST_MAX_ROWS, both head sizes and element types, rows that are nearly dense,
empty, or hold one narrow block."""
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


@pytest.mark.parametrize("D,nk,bn,width,dt", [
    (128, 2400, 128, 2405, torch.bfloat16),     # 307200 gathered tokens in a row: more than 2048 tiles
    (64, 4091, 128, 4096, torch.float16),       # ... and the most a list can hold
    (128, 5000, 32, 1500, torch.bfloat16),      # block numbers above 4095 in lists past the common limit
    (64, 8192, 32, 4096, torch.bfloat16),       # ... up to PSA_FWD_BLOCKS_MAX_ROWS
    (128, 8193, 32, 1500, torch.bfloat16),      # one block more: the scalar kernel takes the call
    (128, 5000, 32, 1472, torch.float16),       # the same in lists up to PSA_FWD_LIST_MAX, row-major ...
    (64, 5000, 64, 700, torch.bfloat16),        # ... and from tile images
    (64, 16384, 32, 1472, torch.bfloat16),      # PSA_FWD_BLOCKS_MAX blocks
    (64, 16385, 64, 300, torch.bfloat16),       # one block more
])
def test_rows_of_very_long_sequences_equal_the_scalar_kernel(D, nk, bn, width, dt):
    from psa_b200 import ops
    S, Sq = nk * bn - 3, 128 + 7
    k, v = (torch.randn((1, 1, S, D), generator=torch.Generator(DEV).manual_seed(810 + i), device=DEV).to(dt) for i in range(2))
    q = C.randn(813, (1, 1, Sq, D), dt).to(DEV)
    room = min(nk, width - 4)
    mask = torch.zeros((1, 1, 2, width), dtype=torch.int32)
    blocks = torch.randperm(nk, generator=torch.Generator().manual_seed(nk)).to(torch.int32)
    blocks[blocks == nk - 1] = blocks[0]
    blocks[0] = nk - 1                                             # the last (ragged) block is among them
    row = blocks[:room].tolist() + [-1] * 4                        # as many level 1 blocks as the list holds
    mask[0, 0, 0, :len(row)] = torch.tensor(row, dtype=torch.int32)
    c = [room // 4, room // 4, room // 4, room - 3 * (room // 4)]   # ... and all four levels
    row = sum((part.tolist() + [-1] for part in blocks[:room].split(c)), [])
    mask[0, 0, 1, :len(row)] = torch.tensor(row, dtype=torch.int32)
    mask = mask.to(DEV)
    auto = ops.psa_forward(q, k, v, mask, 128, bn, 32)
    assert int(auto._psa_status.item()) == 0
    sc = ops.psa_forward(q, k, v, mask, 128, bn, 32, impl=ops.IMPL_SCALAR)
    covered = nk <= (8192 if width > 1472 else 16384)
    if covered:
        tc = ops.psa_forward(q, k, v, mask, 128, bn, 32, impl=ops.IMPL_TENSOR)
        assert int(tc._psa_status.item()) == 0 and torch.equal(auto, tc)
    else:
        assert torch.equal(auto, sc)
        with pytest.raises(ValueError):
            ops.psa_forward(q, k, v, mask, 128, bn, 32, impl=ops.IMPL_TENSOR)
    # a row averages thousands of values: results of 1e-3..1e-2, with the roundings of the test above
    a, b = auto.float(), sc.float()
    assert torch.isfinite(b).all() and float((a - b).norm()) <= 1e-2 * float(b.norm())
