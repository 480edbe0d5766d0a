"""GPU: the antidiagonal estimate of lengths that are no multiple of the stride on the tcgen05 kernel (two pairs of tensor maps)
against the mma.sync kernel, which reads token by token, and the oracle."""
import pytest
import torch

import cases as C
from oracle import psa_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _scratch_used(q, k, block, stride, chunk, causal, impl, want):
    from psa_b200 import _lib, ops
    _, H, L, D = q.shape
    mark = 0x5A5A5A5A
    scratch = torch.full((_lib.lib.psa_antidiag_scratch_bytes(H, L, D, block, stride, chunk) // 4,), mark, dtype=torch.int32, device=DEV)
    out = torch.empty_like(want)
    rc = _lib.lib.psa_antidiag_scores_impl(q.data_ptr(), k.data_ptr(), out.data_ptr(), scratch.data_ptr(), scratch.numel() * 4, H, L, D, block,
                                           stride, chunk, int(causal), ops._dt(q), impl, 0, torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and torch.equal(out, want)
    return scratch != mark


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("L,D,H,block,stride,chunk,causal", [
    (17, 64, 2, 128, 16, 1024, True),        # one whole group and one token
    (31, 128, 1, 128, 16, 1024, False),      # all positions but one have a second group
    (2047, 128, 2, 128, 16, 1024, True),     # last group short of one token, whole row tiles otherwise
    (2049, 64, 3, 128, 16, 1024, True),      # a group row of its own tile for one token
    (1500, 128, 1, 64, 8, 512, False),
    (5003, 128, 2, 128, 16, 2048, True),
])
def test_ragged_lengths(L, D, H, block, stride, chunk, causal, dt):
    from psa_b200 import ops
    q, k, _ = C.qkv(610, 1, H, L, D, dt)
    qd, kd = q.to(DEV), k.to(DEV)
    got = ops.antidiag_block_scores(qd, kd, block, stride, chunk, causal)
    ops.check_status()
    mma = ops.antidiag_block_scores(qd, kd, block, stride, chunk, causal, impl=ops.IMPL_WARP_MMA)
    # the same products accumulated in fp32 by both: one unit in the last place of a 16-bit mass of at most block/stride
    ulp = (block // stride) * 2.0 ** (-8 if dt == torch.bfloat16 else -11)
    assert torch.isfinite(got).all() and float((got.double() - mma.double()).abs().max()) <= ulp
    # ... and by two kernels: each writes other words of the scratch memory (the logits, or the sums of every tile)
    used = [_scratch_used(qd, kd, block, stride, chunk, causal, impl, out) for impl, out in ((0, got), (ops.IMPL_WARP_MMA, mma))]
    assert used[0].any() and used[1].any() and not torch.equal(*used)
    ref = O.antidiag_block_scores(q, k, block, stride, causal, chunk)
    assert float((got.double().cpu() - ref).abs().max()) <= (block // stride) * 2.0 ** -8
