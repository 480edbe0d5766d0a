"""GPU: the layer in one call (psa_layer) against the same kernels called one by one, bit for bit."""
import pytest
import torch

import cases as C

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _same(a, b):
    """Equal bits, a row without a selected block (0/0, as in the reference) included."""
    return torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,Sq,Sk,D,bn,mode", [(1, 2, 1, 1, 64, 64, "topk"), (2, 3, 1000, 1000, 128, 64, "thresholdbound"),
                                                 (1, 2, 300, 2049, 64, 128, "topk"), (2, 1, 4224, 129, 128, 128, "thresholdbound")])
def test_layer_equals_its_kernels(B, H, Sq, Sk, D, bn, mode, dt):
    import psa_b200
    from psa_b200 import ops
    from psa_b200.attention import compute_block_mask
    cfg = psa_b200.PSAConfig(block_n=bn, mask_mode=mode, mask_ratios=C.DEFAULT_RATIOS if mode == "topk" else C.RATIOS_THR)
    q = C.randn(61, (B, H, Sq, D), dt, smooth=8).to(DEV)
    k, v = (C.randn(62 + i, (B, H, Sk, D), dt, smooth=8).to(DEV) for i in range(2))
    k_t = k.transpose(1, 2).contiguous().transpose(1, 2)          # any strides
    iq, ik = C.sample_idx(7, B, H, 128, 32).to(DEV), C.sample_idx(8, B, H, bn, bn // 4).to(DEV)
    assert ops.layer_supported(q, k_t, v, cfg)
    out = psa_b200.PSAAttention(cfg)(q, k_t, v, idx_q=iq, idx_k=ik)
    mask, _, _ = compute_block_mask(q, k, cfg, idx_q=iq, idx_k=ik)
    ref = ops.psa_forward(q, k, v, mask, 128, bn, 32)
    ops.check_status()
    assert out.shape == ref.shape and _same(out, ref)
    torch.manual_seed(3)
    drawn = psa_b200.PSAAttention(cfg)(q, k, v)
    torch.manual_seed(3)
    iq, ik = (ops.draw_sample_indices(B, H, b, b // 4, q.device) for b in (128, bn))
    assert _same(drawn, psa_b200.PSAAttention(cfg)(q, k, v, idx_q=iq.to(torch.int32), idx_k=ik.to(torch.int32)))


def test_other_calls_take_the_single_entry_points():
    import psa_b200
    from psa_b200 import ops
    q = torch.zeros(1, 2, 256, 64, dtype=torch.bfloat16, device=DEV)
    assert ops.layer_supported(q, q, q, psa_b200.PSAConfig())
    assert not ops.layer_supported(q.float(), q.float(), q.float(), psa_b200.PSAConfig())
    assert not ops.layer_supported(q, q, q, psa_b200.PSAConfig(block_n=32))
    assert not ops.layer_supported(q, q[:, :1], q[:, :1], psa_b200.PSAConfig())
    assert not ops.layer_supported(q, q, q, psa_b200.PSAConfig(attn_impl="old_mask_type", block_n=128))
    for mode in ("mass", None):
        cfg = psa_b200.PSAConfig(mask_mode=mode)
        assert not ops.layer_supported(q, q, q, cfg)
        with pytest.raises(ValueError, match=f"Unknown mode: {mode}_newtype"):      # the error of the single entry point
            psa_b200.PSAAttention(cfg)(q, q, q)


def test_an_attention_function_put_in_place_of_the_modules_own_is_called():
    import psa_b200
    from psa_b200 import ops
    from psa_b200.attention import compute_block_mask
    cfg = psa_b200.PSAConfig()
    q, k, v = (x.to(DEV) for x in C.qkv(65, 1, 2, 1500, 64, torch.bfloat16))
    iq, ik = C.sample_idx(9, 1, 2, 128, 32).to(DEV), C.sample_idx(10, 1, 2, 64, 16).to(DEV)
    module = psa_b200.PSAAttention(cfg)
    plain = module(q, k, v, idx_q=iq, idx_k=ik)
    own, calls = module.sparse_attention_fn, []

    def recorded(*args):
        calls.append(args[3].shape)
        return own(*args)
    module.sparse_attention_fn = recorded
    assert _same(module(q, k, v, idx_q=iq, idx_k=ik), plain) and len(calls) == 1
    module.sparse_attention_fn = psa_b200.sparse_attention_factory(128, 32, 64, compat_quirk=False)
    got = module(q, k, v, idx_q=iq, idx_k=ik)
    mask, _, _ = compute_block_mask(q, k, cfg, idx_q=iq, idx_k=ik)
    assert _same(got, ops.psa_forward(q, k, v, mask, 128, 64, 32, compat_quirk=False)) and not _same(got, plain)
    module.sparse_attention_fn = own
    assert _same(module(q, k, v, idx_q=iq, idx_k=ik), plain) and len(calls) == 1
