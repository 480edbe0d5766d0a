"""GPU: the streams of the tcgen05 legacy backward at the sizes where they can go wrong - the dK/dV kernel looks for its query
blocks 32 at a time while a job runs, and the fold deals the positions behind the last token to a block of threads - and an
attention output that is not 16-byte aligned.  Yardstick: the scalar kernels on the same 16-bit inputs."""
import pytest
import torch

import cases as C

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _close(a, b, scale):
    """Both sides round the probabilities and their gradients to 16 bits (8 or 11 significant ones) before the accumulating
    products and the result once more: errors of 2^-8 of the terms, averaging out over a sum.  scale: the norm of dO; a
    gradient that cancels (one key: p = 1, dS = 0) is left with fp32 rounding of the terms."""
    for g, r in zip(a, b):
        g, r = g.double(), r.double()
        assert bool(torch.isfinite(g).all())
        assert float((g - r).norm()) <= 1e-2 * float(r.norm()) + 1e-5 * scale
        assert float((g - r).abs().max()) <= 2e-2 * max(1.0, float(r.abs().max()))


def _run(S, D, dt, causal, mask, o_shift=0):
    from psa_b200 import ops
    B, H = mask.shape[:2]
    q, k, v = (x.to(DEV) for x in C.qkv(520, B, H, S, D, dt))
    do = C.randn(524, (B, H, S, D), dt).to(DEV)
    mask = mask.to(DEV)
    o, lse, kv = ops.legacy_forward(q, k, v, mask, causal, need_lse=True)
    if o_shift:
        o = torch.empty(o.numel() + o_shift, dtype=dt, device=DEV)[o_shift:].copy_(o.flatten()).view(o.shape)
        assert o.data_ptr() % 16 != 0 and o.is_contiguous()
    tc, sc = (ops.legacy_backward(q, k, v, mask, o, lse, do, causal, D ** -0.5, kv, impl=i) for i in (ops.IMPL_TENSOR, ops.IMPL_SCALAR))
    assert int(tc[0]._psa_status.item()) == 0
    _close(tc, sc, float(do.double().norm()))


@pytest.mark.parametrize("causal", [False, True], ids=["full", "causal"])
@pytest.mark.parametrize("S,D,dt", [(128 * 33 + 1, 128, torch.bfloat16), (128 * 32, 64, torch.float16), (128 * 65 - 8, 64, torch.bfloat16),
                                    (128 * 34 - 127, 128, torch.float16)])
def test_more_query_blocks_than_one_search_step(S, D, dt, causal):
    n = -(-S // 128)
    mask = C.legacy_mask(525, 1, 2, S, causal, False)
    lo = 0 if not causal else 1
    mask[0, 0, :32, lo:lo + 1] = 0            # the first 32 query blocks select nothing of this key block ...
    mask[0, 1, 32:, 2:4] = 0                  # ... and none of those behind them anything of these
    mask[0, 1, n - 1] = 0
    mask[0, 1, n - 1, n - 1] = 1              # the last query block reads one block: its own, if causal on the diagonal
    _run(S, D, dt, causal, mask)


@pytest.mark.parametrize("S", [1, 127, 129, 250])
@pytest.mark.parametrize("D", [64, 128])
def test_padded_positions_are_folded_into_the_last_token(S, D):
    mask = C.legacy_mask(526, 1, 2, S, False, False)
    mask[mask == 0] = 4
    _run(S, D, torch.bfloat16, False, mask)


def test_attention_output_need_not_be_aligned():
    _run(300, 128, torch.bfloat16, True, C.legacy_mask(527, 1, 2, 300, True, False), o_shift=1)
