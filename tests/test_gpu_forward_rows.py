"""GPU: the tcgen05 forward at the ends of its rows - rows of 0 to 6 tiles of 128 columns in many orders, so that each softmax group
finishes rows and starts the next ones early, 13 to 22 rows to a CTA (one runs on each of 148 SMs), so that row slots and barriers
go round several times; last tiles of every width; an output that is 16- but not 32-byte aligned, or in the buffers of several
owners; the causal rule, log-sum-exp rows and rows without a visible key; blocks that no row selects and that hold values that are
not finite; first keys far below the rest of the first tile.  Yardstick: the scalar kernel on the same 16-bit inputs."""
import pytest
import torch

import cases as C

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _mask(nk, bn, mq, heads, seed, avoid=()):
    """Rows that select 0 to 6 tiles' worth of blocks, at random levels."""
    g = torch.Generator().manual_seed(seed)
    mask = torch.zeros((1, heads, mq, nk + 5), dtype=torch.int32)
    usable = torch.tensor([b for b in range(nk) if b not in avoid], dtype=torch.int32)
    for h in range(heads):
        for r in range(mq):
            budget = int(torch.randint(0, 7, (1,), generator=g)) * 128 - int(torch.randint(0, 128, (1,), generator=g))
            blocks = usable[torch.randperm(len(usable), generator=g)].tolist()
            share = torch.rand(4, generator=g) * (torch.rand(4, generator=g) < 0.7)
            row, at = [], 0
            for li in range(4):
                n = max(0, int(budget * float(share[li]) / max(1e-6, float(share.sum())) / (bn >> li)))
                n = min(n, len(blocks) - at)
                row += blocks[at:at + n] + [-1]
                at += n
            mask[0, h, r, :len(row)] = torch.tensor(row, dtype=torch.int32)
    return mask.to(DEV)


def _close(a, b):
    """Probabilities and results rounded to 8 (bf16) or 11 bits by both; a probability relative to another reference rounds anew."""
    a, b = a.float(), b.float()
    assert torch.equal(torch.isnan(a), torch.isnan(b))
    a, b = a.nan_to_num(), b.nan_to_num()
    assert float((a - b).abs().max()) <= 2e-2 * max(1.0, float(b.abs().max())) and float((a - b).norm()) <= 1e-2 * float(b.norm())


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("D,bn", [(128, 64), (64, 64), (128, 128), (64, 128), (128, 32), (64, 32)])
def test_short_rows_in_every_order(D, bn, dt):
    from psa_b200 import ops
    heads, mq, nk = 48, 70, 1024 // bn + 9
    S = nk * bn - 3
    k, v = (C.randn(900 + i, (1, heads, S, D), dt).to(DEV) for i in range(2))
    q = C.randn(903, (1, heads, mq * 128 - 5, D), dt).to(DEV)
    mask = _mask(nk, bn, mq, heads, 10 * bn + D)
    out = torch.full((q.numel() + 8,), 7.0, dtype=dt, device=DEV)[8:].view(q.shape)
    assert out.data_ptr() % 32 == 16
    tc = ops.psa_forward(q, k, v, mask, 128, bn, 32, out=out)
    assert int(tc._psa_status.item()) == 0
    sc = ops.psa_forward(q, k, v, mask, 128, bn, 32, impl=ops.IMPL_SCALAR)
    _close(tc, sc)
    again = ops.psa_forward(q, k, v, mask, 128, bn, 32)
    assert again.data_ptr() % 32 == 0
    assert torch.equal(again.nan_to_num(), tc.nan_to_num())
    _close(again, sc)


@pytest.mark.parametrize("bn", [32, 64, 128])
def test_blocks_that_no_row_selects_may_hold_anything(bn):
    from psa_b200 import ops
    heads, mq, nk, D = 48, 40, 1024 // bn + 9, 128
    S = nk * bn
    bad = (0, 2, 3, 5)      # block 0 and those that narrow levels pair up with (2, 3 at most)
    k, v = (C.randn(910 + i, (1, heads, S, D), torch.bfloat16).to(DEV) for i in range(2))
    q = C.randn(913, (1, heads, mq * 128, D), torch.bfloat16).to(DEV)
    mask = _mask(nk, bn, mq, heads, bn, avoid=bad)
    clean = ops.psa_forward(q, k, v, mask, 128, bn, 32, compat_quirk=False)
    for b, x in zip(bad, (float("inf"), float("nan"), float("-inf"), float("inf"))):
        k[:, :, b * bn:(b + 1) * bn] = x
        v[:, :, b * bn:(b + 1) * bn] = x
    dirty = ops.psa_forward(q, k, v, mask, 128, bn, 32, compat_quirk=False)
    assert torch.equal(torch.nan_to_num(clean.float(), nan=3.0), torch.nan_to_num(dirty.float(), nan=3.0))


@pytest.mark.parametrize("D", [64, 128])
def test_first_keys_far_below_the_rest_of_the_first_tile(D):
    from psa_b200 import ops
    nk, bn, heads = 8, 64, 2
    S = nk * bn
    q, k, v = (C.randn(920 + i, (1, heads, S, D), torch.bfloat16).to(DEV) for i in range(3))
    for octaves in (20, 300):      # inside the range that one reference covers, and past it
        q[..., 0] = 16.0
        k[..., 0] = 0.0
        k[:, :, :32, 0] = -octaves * 0.6931 * D ** 0.5 / 16.0
        mask = torch.zeros((1, heads, S // 128, nk + 5), dtype=torch.int32, device=DEV)
        mask[..., :nk] = torch.arange(nk, device=DEV, dtype=torch.int32)
        mask[..., nk:nk + 4] = -1
        tc = ops.psa_forward(q, k, v, mask, 128, bn, 32)
        sc = ops.psa_forward(q, k, v, mask, 128, bn, 32, impl=ops.IMPL_SCALAR)
        assert int(tc._psa_status.item()) == 0
        _close(tc, sc)


@pytest.mark.parametrize("empty", [0.97, 0.6])
def test_rows_without_tiles_among_others(empty):
    """Most rows select no block (0/0, as the reference divides) - runs of them hand the four row slots of a CTA round and round,
    about 22 rows per CTA; the others select one to three tiles."""
    from psa_b200 import ops
    heads, mq, nk, bn, D = 48, 70, 25, 64, 64
    k, v = (C.randn(930 + i, (1, heads, nk * bn, D), torch.bfloat16).to(DEV) for i in range(2))
    q = C.randn(933, (1, heads, mq * 128, D), torch.bfloat16).to(DEV)
    g = torch.Generator().manual_seed(int(empty * 100))
    level = torch.randint(0, 4, (heads, mq), generator=g)
    count = torch.randint(1, 7, (heads, mq), generator=g) * (torch.rand(heads, mq, generator=g) >= empty)
    mask = torch.full((1, heads, mq, nk + 5), -1, dtype=torch.int32)
    for h in range(heads):
        for r in range(mq):
            n, at = int(count[h, r]), int(level[h, r])      # `at` empty levels before the one that holds the row's blocks
            mask[0, h, r, at:at + n] = torch.randperm(nk, generator=g)[:n].to(torch.int32)
    mask = mask.to(DEV)
    tc = ops.psa_forward(q, k, v, mask, 128, bn, 32)
    assert int(tc._psa_status.item()) == 0
    rows_nan = torch.isnan(tc.float()).view(heads, mq, 128 * D)
    assert torch.equal(rows_nan.all(-1).cpu(), count == 0) and torch.equal(rows_nan.any(-1).cpu(), count == 0)
    _close(tc, ops.psa_forward(q, k, v, mask, 128, bn, 32, impl=ops.IMPL_SCALAR))
    again = ops.psa_forward(q, k, v, mask, 128, bn, 32)
    assert torch.equal(tc.nan_to_num(), again.nan_to_num())


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("D,bn,images", [(128, 64, True), (64, 64, True), (128, 64, False), (64, 64, False), (128, 32, False), (64, 32, False)])
def test_infinite_value_in_the_last_selected_block(D, bn, images, dt):
    """A selected value that is infinite makes its channel infinite, not NaN, however the row's last tile is filled up: rows that end
    in a block of 4 or 8 columns, one to four tiles long, the last block the one with the infinite value."""
    from psa_b200 import ops
    heads, mq, nk = 2, 40, 1024 // bn + 9
    S = nk * bn
    k, v = (C.randn(940 + i, (1, heads, S, D), dt).to(DEV) for i in range(2))
    q = C.randn(943, (1, heads, mq * 128, D), dt).to(DEV)
    v[0, :, S - bn + 5, 3], v[0, :, S - bn + 5, 7] = float("inf"), float("-inf")
    mask = torch.full((1, heads, mq, nk + 5), -1, dtype=torch.int32)
    for r in range(mq):
        n = 1 + r % (nk - 1)            # blocks of level 1 before the last block of the sequence at level 8
        mask[:, :, r, :n] = torch.arange(n, dtype=torch.int32)
        mask[:, :, r, n + 3] = nk - 1
    mask = mask.to(DEV)
    tc = ops.psa_forward(q, k, v, mask, 128, bn, 32, pyramid=None if images else ops.pyramid_kv(k, v, bn))
    assert int(tc._psa_status.item()) == 0
    assert bool((tc[..., 3] == float("inf")).all()) and bool((tc[..., 7] == float("-inf")).all())
    sc = ops.psa_forward(q, k, v, mask, 128, bn, 32, impl=ops.IMPL_SCALAR)
    keep = [c for c in range(D) if c not in (3, 7)]
    assert bool(torch.isfinite(tc[..., keep]).all())
    _close(tc[..., keep], sc[..., keep])


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True], ids=["full", "causal"])
def test_bf16_reference_is_the_maximum_of_the_whole_first_tile(D, causal):
    """96 of a tile's 128 keys stand 0.3 octaves above the first 32 and alone carry values.  Relative to the tile's maximum their
    probabilities are exactly 1 and the result is right but for its own rounding, up to 2^-9 either way, which averages out over
    the channels to a few 1e-4; relative to the first 32 keys all of them round by the same 2.5e-3."""
    from psa_b200 import ops
    S, tokens = 256, 128
    k0 = 0.3 * 0.693147 * D ** 0.5
    q, k, v = (torch.zeros((1, 1, S, D), dtype=torch.float64) for _ in range(3))
    q[..., 0] = 1.0
    k[0, 0, 32:128, 0] = k0
    v[0, 0, 32:128] = 1.0 + torch.arange(D, dtype=torch.float64) / D
    q, k, v = (x.to(torch.bfloat16) for x in (q, k, v))
    p = torch.exp((q.double() @ k[:, :, :tokens].double().transpose(2, 3)) * D ** -0.5)
    want = (p @ v[:, :, :tokens].double() / p.sum(-1, keepdim=True))[:, :, 128:]     # rows that see all of the first 128 keys
    if causal:
        mask = torch.tensor([[1, 0], [1, 0]], dtype=torch.int32).view(1, 1, 2, 2)
        out, _, _ = ops.legacy_forward(q.to(DEV), k.to(DEV), v.to(DEV), mask.to(DEV), True)
    else:
        mask = torch.tensor([0, 1, -1, -1, -1, -1, 0, 0], dtype=torch.int32).view(1, 1, 1, 8).expand(1, 1, 2, 8).contiguous()
        out = ops.psa_forward(q.to(DEV), k.to(DEV), v.to(DEV), mask.to(DEV), 128, 64, 32)
    assert int(out._psa_status.item()) == 0
    got = out[:, :, 128:].double().cpu()
    assert abs(float((got / want).mean()) - 1.0) <= 1e-3


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("D,bn", [(64, 64), (128, 64), (64, 32), (128, 32)])
def test_large_equal_scores_in_a_tile_that_ends_early(D, bn, dt):
    """Equal scores of 2^17 to 2^19 octaves (half of that in fp16) in a tile of 4 or 8 columns: the reference is one of them, so every
    probability is exactly 1 and the result the common value.  A score that is multiplied by the scale and reduced by the rounded
    reference in one step leaves what the reference's rounding took, up to half a unit of 2^-5 octaves, in the sum but not in the
    rounded probabilities."""
    from psa_b200 import ops
    unit = 1.0 if dt == torch.bfloat16 else 0.5
    gains = [129, 131, 133, 137, 139, 143]
    heads, S = len(gains), 8 * bn
    q = torch.full((1, heads, 256, D), 128.0 * unit)
    k = torch.tensor(gains, dtype=torch.float32).view(1, heads, 1, 1).expand(1, heads, S, D).contiguous()
    v = torch.ones((1, heads, S, D))
    q, k, v = (x.to(dt).to(DEV) for x in (q, k, v))
    assert k.float().mean(dim=(2, 3)).cpu().view(-1).tolist() == gains
    mask = torch.tensor([-1, -1, -1, 3, -1] + [0] * 8, dtype=torch.int32).view(1, 1, 1, 13).expand(1, heads, 2, 13).contiguous().to(DEV)
    out = ops.psa_forward(q, k, v, mask, 128, bn, 32)
    assert int(out._psa_status.item()) == 0
    assert bool((out == 1).all()), out[0, :, 0, 0].tolist()


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [False, True], ids=["full", "causal"])
def test_short_rows_of_the_old_format(D, causal, dt):
    """Rows of 0 to 6 tiles from level masks, with log-sum-exp: rows without a block or (causal, diagonal block of a pooled level alone)
    without a visible key give 0 and -inf; a last block that ends inside a group of four columns."""
    from psa_b200 import ops
    heads, nb = 48, 70
    S = nb * 128 - 5
    q, k, v = (C.randn(950 + i, (1, heads, S, D), dt).to(DEV) for i in range(3))
    g = torch.Generator().manual_seed(D + causal)
    mask = torch.zeros((1, heads, nb, nb), dtype=torch.int32)
    levels = torch.tensor([1, 2, 4, 8], dtype=torch.int32)
    for h in range(heads):
        for m in range(nb):
            seen = m + 1 if causal else nb
            n = min(int(torch.randint(0, 7, (1,), generator=g)), seen)
            picks = torch.randperm(seen, generator=g)[:n]
            if n and int(torch.randint(0, 2, (1,), generator=g)):
                picks[0] = seen - 1                       # the diagonal block, or the sequence's last one
            mask[0, h, m, picks] = levels[torch.randint(0, 4, (n,), generator=g)]
    mask = mask.to(DEV)
    out, lse, _ = ops.legacy_forward(q, k, v, mask, causal, need_lse=True)
    assert int(out._psa_status.item()) == 0
    ref, ref_lse, _ = ops.legacy_forward(q, k, v, mask, causal, need_lse=True, impl=ops.IMPL_SCALAR)
    _close(out, ref)
    dead = torch.isinf(ref_lse)
    assert bool(dead.any()) and torch.equal(dead, torch.isinf(lse)) and bool((lse[dead] < 0).all()) and bool((out[dead] == 0).all())
    # fp32 sums of at most 768 terms in another order, and an exp2 that is right to 2^-22
    assert float((lse[~dead] - ref_lse[~dead]).abs().max()) <= 1e-4
    again, lse2, _ = ops.legacy_forward(q, k, v, mask, causal, need_lse=True)
    assert torch.equal(out, again) and torch.equal(lse, lse2)


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("D,bn,owners", [(128, 64, 2), (64, 128, 3)])
def test_rows_scattered_to_several_owners(D, bn, owners, dt):
    """Output rows that go to the buffer of the rank that owns the token, all of them in this GPU's memory here: the bits of the plain
    forward at the places of the address contract, nothing anywhere else."""
    import ctypes
    from psa_b200 import ops
    from psa_b200._lib import check, lib
    heads, head0, total, mq, nk = 6, 3, 11, 70, 1024 // bn + 9
    S, Sq = nk * bn - 3, mq * 128 - 5
    per = -(-Sq // owners)
    k, v = (C.randn(960 + i, (1, heads, S, D), dt).to(DEV) for i in range(2))
    q = C.randn(963, (1, heads, Sq, D), dt).to(DEV)
    mask = _mask(nk, bn, mq, heads, 7 * bn)
    images = ops.pyramid_kv_images(k, v, bn)
    want = ops.psa_forward(q, k, v, mask, 128, bn, 32, pyramid=images)
    bufs = [torch.full((per, total, D), 7.0, dtype=dt, device=DEV) for _ in range(owners)]
    peers = (ctypes.c_void_p * owners)(*[b.data_ptr() for b in bufs])
    status = ops.status_word(q.device)
    check(lib.psa_fwd_images_scatter(q.data_ptr(), images.kimg.data_ptr(), images.vimg.data_ptr(), mask.data_ptr(), peers, owners, per, total,
                                     head0, heads, Sq, S, D, 128, bn, 32, mask.shape[-1], D ** -0.5, 1, ops._dt(q), status.data_ptr(),
                                     ops._stream(q)), "psa_fwd_images_scatter")
    assert int(status.item()) == 0
    got = torch.cat(bufs)
    assert torch.equal(got[:Sq, head0:head0 + heads].transpose(0, 1).nan_to_num(), want[0].nan_to_num())
    got[:Sq, head0:head0 + heads] = 7.0
    assert bool((got == 7.0).all())
