"""GPU: q, k, v laid out by one kernel (order, rotation, caller's strides) against the framework's element-wise operations,
and the module's routes that use it against the same route on operands prepared with those operations - bit for bit."""
import pytest
import torch

import cases as C

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _tables(S, first, D):
    from psa_b200 import ops
    ang = torch.rand(S - first, D, generator=torch.Generator().manual_seed(3)) * 6.28
    return ops.RotaryTables(torch.cos(ang).to(DEV), torch.sin(ang).to(DEV), first)


def _layout(x, kind):
    """The same values [B, H, S, D] under other strides."""
    if kind == "token":
        return x.transpose(1, 2).contiguous().transpose(1, 2)
    if kind == "fused":       # a slice of one projection's output [B, S, 3, H, D]
        B, H, S, D = x.shape
        y = torch.zeros((B, S, 3, H, D), dtype=x.dtype, device=x.device)
        y[:, :, 1] = x.transpose(1, 2)
        return y[:, :, 1].transpose(1, 2)
    if kind == "odd":         # strides and start that are no multiple of 16 bytes
        y = torch.zeros((*x.shape[:3], x.shape[3] + 3), dtype=x.dtype, device=x.device)
        y[..., 3:] = x
        return y[..., 3:]
    if kind == "channel":     # channels not contiguous
        return x.transpose(2, 3).contiguous().transpose(2, 3)
    return x


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,S,D,first", [(1, 3, 1000, 128, 0), (2, 2, 65, 64, 17), (1, 1, 1, 128, 0), (2, 5, 257, 64, 257)])
@pytest.mark.parametrize("kinds", [("head", "head", "token"), ("token", "fused", "odd"), ("channel", "token", "head")])
def test_views_equal_elementwise_copies(kinds, B, H, S, D, first, dt):
    from psa_b200 import ops
    x = [C.randn(30 + i, (B, H, S, D), dt).to(DEV) for i in range(3)]
    rope = _tables(S, first, D)
    perm = torch.randperm(S, generator=torch.Generator().manual_seed(5)).to(torch.int32).to(DEV)
    views = [_layout(a, k) for a, k in zip(x, kinds)]
    for p in (None, perm):
        for r in (None, rope):
            want = [ops.rotate_rows(a, r) if r is not None and i < 2 else a for i, a in enumerate(x)]
            want = want if p is None else [a[:, :, p.long()] for a in want]
            assert ops.views_supported(*views, r)
            for got, ref in zip(ops.gather_views(*views, p, r), want):
                assert got.is_contiguous() and torch.equal(got, ref)


@pytest.mark.parametrize("impl,bn,rearrange,mode,text", [("old_mask_type", 128, True, "thresholdbound", 0), ("new_mask_type", 32, True, "topk", 20),
                                                         ("new_mask_type", 64, False, "topk", 20), ("old_mask_type", 128, False, "topk", 0)])
@pytest.mark.parametrize("kinds", [("token",) * 3, ("head", "head", "token")])
def test_module_routes_equal_rotated_copies(kinds, impl, bn, rearrange, mode, text):
    from psa_b200 import ops
    from psa_b200.pyramid_sparse_attention import AttentionConfig, PyramidSparseAttention
    W, Hh, T, H, D = 12, 8, 9, 2, 128
    cfg = AttentionConfig(width=W, height=Hh, depth=T, text_length=text, use_rearrange=rearrange, rearrange_method="Gilbert",
                          block_m=128, block_n=bn, tile_n=32, use_sim_mask=impl == "old_mask_type",
                          mask_ratios=C.DEFAULT_RATIOS if mode == "topk" else C.RATIOS_THR, mask_mode=mode,
                          warmup_steps=0, attn_impl=impl, sim_2x_threshold=0.7, sim_4x_threshold=0.65, sim_8x_threshold=0.6)
    mod = PyramidSparseAttention(cfg, inference_num=10, layer_num=1, model_type="cogvideo")
    S = W * Hh * T + text
    q, k, v = (_layout(x.to(DEV), kind) for x, kind in zip(C.qkv(981, 1, H, S, D, torch.bfloat16, smooth=16), kinds))
    rope = _tables(S, text, D)
    torch.manual_seed(21)
    fused = mod(q, k, v, 0, rotary=rope)
    torch.manual_seed(21)
    plain = mod(ops.rotate_rows(q, rope), ops.rotate_rows(k, rope), v.contiguous(), 0)
    ops.check_status()
    assert fused.shape == plain.shape and fused.stride() == plain.stride()
    assert torch.equal(fused, plain)


def test_what_the_copy_kernel_does_not_take_goes_the_old_way():
    from psa_b200 import ops
    q, k, v = (C.randn(40 + i, (1, 2, 64, 64), torch.bfloat16).to(DEV) for i in range(3))
    assert ops.views_supported(q, k, v) and not ops.views_supported(q.float(), k.float(), v.float())
    assert not ops.views_supported(q, k, v[:, :, :32]) and not ops.views_supported(q.requires_grad_(), k, v)
    with torch.no_grad():
        assert ops.views_supported(q, k, v) and not ops.views_supported(q, k, v, _tables(65, 0, 64))


def test_an_attention_function_put_in_place_of_the_modules_own_is_called():
    from psa_b200.pyramid_sparse_attention import AttentionConfig, PyramidSparseAttention
    cfg = AttentionConfig(width=12, height=8, depth=9, text_length=20, use_rearrange=True, rearrange_method="Gilbert", block_m=128, block_n=32,
                          tile_n=32, use_sim_mask=False, mask_ratios=C.DEFAULT_RATIOS, mask_mode="topk", warmup_steps=0,
                          attn_impl="new_mask_type")
    mod = PyramidSparseAttention(cfg, inference_num=10, layer_num=1, model_type="cogvideo")
    S = 12 * 8 * 9 + 20
    q, k, v = (_layout(x.to(DEV), "token") for x in C.qkv(982, 1, 2, S, 128, torch.bfloat16, smooth=16))
    rope = _tables(S, 20, 128)
    torch.manual_seed(22)
    plain = mod(q, k, v, 0, rotary=rope)
    own, calls = mod.sparse_attention_fn, []

    def negated(*args):
        calls.append(args[3].shape)
        return -own(*args)
    mod.sparse_attention_fn = negated
    torch.manual_seed(22)
    assert torch.equal(mod(q, k, v, 0, rotary=rope), -plain) and len(calls) == 1
