"""GPU: the scalar forward when a call is small enough that the rows of a query block and the chunks of a row are dealt to several
sets of threads, against the oracle: one chunk only, chunk counts that do not divide, blocks narrower than a chunk, empty rows,
both head sizes, and a call large enough to take no split."""
import pytest
import torch

import cases as C
from oracle import psa_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("B,H,S,D,bm,bn", [(1, 1, 40, 64, 128, 64), (1, 2, 700, 128, 128, 128), (1, 1, 1300, 64, 64, 32), (2, 1, 900, 64, 32, 64),
                                           (1, 3, 513, 128, 128, 32), (4, 24, 300, 64, 128, 64)])
def test_split_rows_and_chunks(B, H, S, D, bm, bn):
    from psa_b200 import ops
    q, k, v = C.qkv(710, B, H, S, D, torch.float32)
    mq, nk = -(-S // bm), -(-S // bn)
    po = C.scores_like(711, B, H, mq, nk, torch.float32)
    mask = O.assign_levels(po, C.DEFAULT_RATIOS, "topk_newtype", bn, 32)
    mask[0, 0, mq - 1, :] = 0
    mask[0, 0, mq - 1, :4] = -1                                   # a row that selects nothing: 0/0
    mask[0, 0, 0, :] = 0
    mask[0, 0, 0, :5] = torch.tensor([nk - 1, -1, -1, -1, -1])      # a row with one block
    out = ops.psa_forward(*(x.to(DEV) for x in (q, k, v)), mask.to(DEV), bm, bn, 32).cpu()
    ref = O.psa_forward_newmask(q, k, v, mask, bm, bn, 32)
    assert torch.equal(torch.isnan(out), torch.isnan(ref))
    # fp32 sums of at most a few thousand terms in another order
    assert float((out - ref).nan_to_num().norm()) <= 1e-5 * float(ref.nan_to_num().norm())
