"""GPU: level assignment of 16-bit scores at the row lengths where its sort changes shape (whole and partial 32-element steps
of the eight warps, each unrolled size, the longest row it takes and the first one past it), bit-exact against the oracle."""
import numpy as np
import pytest
import torch

import cases as C
from oracle import psa_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("nk", [2, 31, 33, 255, 256, 257, 512, 513, 1280, 1281, 1536, 1537, 2048, 2049, 3072, 3073, 4095, 4096, 4097])
@pytest.mark.parametrize("dt,mode", [(torch.bfloat16, "topk_newtype"), (torch.float16, "thresholdbound_newtype"),
                                     (torch.bfloat16, "thresholdbound"), (torch.float32, "thresholdbound")])
def test_row_lengths(nk, dt, mode):
    from psa_b200 import ops
    po = C.scores_like(nk, 1, 2, 3, nk, dt, ties=True)
    ratios = C.RATIOS_THR if mode.startswith("threshold") else C.DEFAULT_RATIOS
    mask = ops.assign_levels(po.to(DEV), ratios, mode, 64, 32)
    assert torch.equal(mask.cpu(), O.assign_levels(po, ratios, mode, 64, 32))


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_signs_zeros_infinities_and_equal_scores(dt):
    """Every order the key mapping has to get right: negative scores, both zeros (equal), infinities, long runs of one value."""
    from psa_b200 import ops
    rng = np.random.default_rng(4)
    vals = torch.tensor([-np.inf, -2.0, -0.0, 0.0, 1e-7, 0.5, 0.5, 3.0, np.inf])
    po = vals[torch.from_numpy(rng.integers(0, vals.numel(), size=(1, 2, 4, 700)))].to(dt)
    mask = ops.assign_levels(po.to(DEV), C.DEFAULT_RATIOS, "topk_newtype", 64, 32)
    assert torch.equal(mask.cpu(), O.assign_levels(po, C.DEFAULT_RATIOS, "topk_newtype", 64, 32))
