"""The calls that the library's speed is judged by: what each of them stands for, its inputs, one pass, its work.

Every case is one attention call through a public entry point, on tensors as the surrounding model holds them:

  module   PSAAttention(config)(q, k, v) on head-major tensors, any block size, mask mode and element type
  preset   PyramidSparseAttention set up by a preset of attention_config.yaml, called as the video models' attention
           processors call it: the Wan processors hand over transposed views of [B, S, H, D] projections, the CogVideoX
           one head-major q and k (its norms are per head) and a transposed view of v; both with their rotary tables
  train    the differentiable kernel of the old mask format, causal: forward and all three gradients
  causal   the vision-language call site (estimate, level mask, similarity cap, causal attention), as prefill or as a
           training step

Run from the repository's root.
"""
import math
import os
import sys

import numpy as np
import torch

_PACKAGE = os.path.join(os.getcwd(), "pyramid-sparse-attention_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(1, _PACKAGE)

import psa_b200
from psa_b200 import ops
from psa_b200.causal import AttentionConfig as CausalConfig
from psa_b200.causal import PyramidAdaptiveBlockSparseAttnTrain
from psa_b200.presets import WanAttentionConfigLoader
from psa_b200.pyramid_sparse_attention import AttentionConfig, PyramidSparseAttention
from psa_b200.synthetic import structured_field

DEVICE = "cuda:0"
DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}

# rank ranges of the levels: the library's defaults (about 15 % of the keys are read) and the 90 % setting of the benchmark
RATIOS = {
    "default": {1: (0.0, 0.1), 2: (0.1, 0.15), 4: (0.15, 0.15), 8: (0.15, 0.35), 0: (0.35, 1.0)},
    "sparse90": {1: (0.0, 0.05), 2: (0.05, 0.1), 4: (0.1, 0.15), 8: (0.15, 0.25), 0: (0.25, 1.0)},
    # cumulative mass instead of rank
    "mass": {1: (0.0, 0.5), 2: (0.5, 0.6), 4: (0.6, 0.7), 8: (0.7, 0.8), 0: (0.8, 1.0)},
}

# model -> (heads, head_dim, [video shapes width x height x frames])
MODELS = {
    "Wan2.1_1.3b": (12, 128, [(832, 480, 81)]),
    "Wan2.1_14b": (40, 128, [(832, 480, 81), (1280, 720, 81)]),
    "Wan2.2_A14B": (40, 128, [(832, 480, 81), (1280, 720, 81)]),
    "Wan2.2_5B": (24, 128, [(1280, 704, 121)]),
    "CogVideo_5b": (48, 64, [(720, 480, 49)]),
    "CogVideo1.5_5b": (48, 64, [(1360, 768, 81)]),
}
PRESETS = [("Wan2.1_1.3b", "psa_balanced"), ("Wan2.1_1.3b", "psa_topk"), ("Wan2.1_14b", "psa_balanced"),
           ("Wan2.2_A14B", "psa_balanced"), ("Wan2.2_5B", "psa_balanced"), ("CogVideo_5b", "psa_balanced"),
           ("CogVideo_5b", "psa_4steps"), ("CogVideo1.5_5b", "psa_balanced")]
# share of the keys that is read (a pooled token counts once) where it depends on the inputs, as measured on these ones:
# cumulative-mass selections, and the causal site, whose similarity cap and text rows refine what the ranks select.
# Plain rank selections follow from their ranges.
MASS_DENSITY = {"Wan2.1_1.3b": 0.67, "Wan2.1_14b": 0.36, "Wan2.2_A14B": 0.40, "Wan2.2_5B": 0.475, "module": 0.45}
CAUSAL_DENSITY = 0.45


def listed():
    return [
        # the smallest calls: a clip of 4096 tokens in fp32 with the default settings ...
        dict(name="module-4k-f32", kind="module", dtype="f32", batch=1, heads=2, tokens=4096, head_dim=64, block_n=64,
             mode="topk", ratios="default"),
        # ... and a single latent frame (one image) of the small video model, where launches and host work count
        dict(name="module-frame", kind="module", dtype="bf16", batch=1, heads=12, tokens=1560, head_dim=128, block_n=64,
             mode="topk", ratios="sparse90"),
        # one self-attention layer of the small and of the large video model (the benchmark's shapes)
        dict(name="module-1.3b", kind="module", dtype="bf16", batch=1, heads=12, tokens=32760, head_dim=128, block_n=64,
             mode="topk", ratios="sparse90"),
        dict(name="module-14b", kind="module", dtype="bf16", batch=1, heads=40, tokens=75600, head_dim=128, block_n=64,
             mode="topk", ratios="sparse90"),
        # fp16, two samples (classifier-free guidance in one batch), a ragged token count
        dict(name="module-ragged-f16", kind="module", dtype="f16", batch=2, heads=16, tokens=9973, head_dim=64, block_n=64,
             mode="topk", ratios="default"),
        # the presets as the processors call them: default of the small Wan model (old mask format, similarity cap,
        # Gilbert order), default of the large one at 480p (separator format, blocks of 128, Gilbert order), the preset with
        # blocks of 32, and the CogVideoX one (text tokens, no reordering)
        dict(name="preset-wan2.1-1.3b", kind="preset", dtype="bf16", model="Wan2.1_1.3b", preset="psa_balanced", width=832,
             height=480, frames=81, heads=12),
        dict(name="preset-wan2.1-14b", kind="preset", dtype="bf16", model="Wan2.1_14b", preset="psa_balanced", width=832,
             height=480, frames=81, heads=40),
        dict(name="preset-wan2.2-5b", kind="preset", dtype="bf16", model="Wan2.2_5B", preset="psa_balanced", width=1280,
             height=704, frames=121, heads=24),
        dict(name="preset-cogvideox-5b", kind="preset", dtype="bf16", model="CogVideo_5b", preset="psa_balanced", width=720,
             height=480, frames=49, heads=48),
        # a training step of the causal kernels at the benchmark's size
        dict(name="train-causal-32k", kind="train", dtype="bf16", batch=2, heads=16, tokens=32768, head_dim=128),
        # vision-language prefill at the benchmark's size, and a training step on a prompt of ordinary, ragged length
        dict(name="causal-prefill-32k", kind="causal", dtype="bf16", heads=28, tokens=32768, train=False),
        dict(name="causal-train-ragged", kind="causal", dtype="bf16", heads=28, tokens=5003, train=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    known = [{k: v for k, v in case.items() if k != "name"} for case in listed()]
    case = _draw(rng)
    while case in known:
        case = _draw(rng)
    return case


def _draw(rng):
    kind = rng.choice(["module", "module", "module", "preset", "preset", "train", "causal"])
    if kind == "module":
        dtype = rng.choice(["bf16"] * 6 + ["f16"] * 3 + ["f32"])
        head_dim, block_n = rng.choice([64, 128]), rng.choice([32, 64, 64, 64, 128])
        # fp32 stands for checks and small experiments; blocks of 32 tokens for the clips of the presets that use them
        tokens = _log_int(rng, 1024, 6000 if dtype == "f32" else 47000 if block_n == 32 else 75600)
        batch = rng.choice([1, 1, 2]) if tokens < 20000 else 1
        budget = 2 * 4096 ** 2 * 64 if dtype == "f32" else 40 * 75600 ** 2 * 128 // 4
        heads = max(1, min(rng.randint(1, 48), int(budget // (batch * tokens ** 2 * head_dim))))
        return dict(kind=kind, dtype=dtype, batch=batch, heads=heads, tokens=tokens, head_dim=head_dim, block_n=block_n,
                    mode="topk" if dtype == "f32" or rng.random() < 0.7 else "thresholdbound", ratios=rng.choice(["default", "sparse90"]))
    if kind == "preset":
        model, preset = rng.choice(PRESETS)
        heads, _, shapes = MODELS[model]
        width, height, frames = rng.choice(shapes)
        # clips come shorter than the model's longest, and heads are sharded over 1 to 8 GPUs (at 720p a layer of the large
        # models is the work of several GPUs)
        case = dict(kind=kind, dtype=rng.choice(["bf16", "bf16", "f16"]), model=model, preset=preset, width=width, height=height,
                    frames=4 * rng.randint(4, (frames - 1) // 4) + 1)
        share = rng.choice([1, 2, 4])
        while heads // share * _preset_tokens(case) ** 2 > 1.1 * 40 * 32760 ** 2:
            share *= 2
        return dict(case, heads=heads // share)
    if kind == "train":
        return dict(kind=kind, dtype=rng.choice(["bf16", "bf16", "f16"]), batch=rng.choice([1, 2]), heads=rng.randint(2, 16),
                    tokens=_log_int(rng, 1024, 32768), head_dim=rng.choice([64, 128]))
    return dict(kind=kind, dtype=rng.choice(["bf16", "bf16", "f16"]), heads=rng.choice([12, 16, 28]),
                tokens=_log_int(rng, 1500, 32768), train=rng.random() < 0.5)


# ------------------------------------------------------------------------------------------------ inputs
def _grid(tokens):
    """Frames x height x width of a clip of at least `tokens` tokens (the last ones are cut off)."""
    side = max(1, int(round(tokens ** (1.0 / 3.0))))
    return (-(-tokens // (side * side)), side, side)


def _fields(seed, batch, heads, tokens, head_dim, dtype, grid=None, text=0):
    """q, k, v [batch, heads, tokens, head_dim]: smooth random fields over the clip plus noise."""
    grid = grid or _grid(tokens)
    return [torch.cat([structured_field(seed * 64 + 8 * b + i, heads, head_dim, grid, text, dtype, DEVICE,
                                        token_range=(0, tokens)) for b in range(batch)]) for i in range(3)]


def _rotary(tokens, head_dim, first):
    """cos / sin tables [tokens - first, head_dim], each value standing twice (channel pairs turn together)."""
    freq = 1.0 / 10000.0 ** (torch.arange(0, head_dim, 2, device=DEVICE, dtype=torch.float32) / head_dim)
    angle = torch.arange(tokens - first, device=DEVICE, dtype=torch.float32)[:, None] * freq[None, :]
    return ops.RotaryTables(angle.cos().repeat_interleave(2, 1), angle.sin().repeat_interleave(2, 1), first)


def _preset(case):
    info = WanAttentionConfigLoader().get_attention_config(case["model"], case["preset"], (case["width"], case["height"], case["frames"]))
    params = dict(info["params"], warmup_steps=0, verbose=False)   # a step after the dense warm-up
    return AttentionConfig(**params)


def _preset_tokens(case):
    c = _preset(case)
    return c.width * c.height * c.depth + c.text_length


def _random_level_mask(seed, batch, heads, tokens):
    n = -(-tokens // 128)
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    weights = torch.tensor([0.2, 0.3, 0.2, 0.15, 0.15], device=DEVICE)
    levels = torch.tensor([0, 1, 2, 4, 8], dtype=torch.int32, device=DEVICE)
    pick = torch.multinomial(weights, batch * heads * n * n, replacement=True, generator=g) if batch * heads * n * n <= 1 << 23 else \
        torch.cat([torch.multinomial(weights, heads * n * n, replacement=True, generator=g) for _ in range(batch)])
    mask = levels[pick].view(batch, heads, n, n)
    mask[..., 0] = 1
    return torch.tril(mask)


def prepare(case, seed):
    torch.manual_seed(seed)          # the sample offsets of the calls come from torch's generator
    kind, dtype = case["kind"], DTYPES[case["dtype"]]
    state = dict(kind=kind)
    if kind == "module":
        state["q"], state["k"], state["v"] = _fields(seed, case["batch"], case["heads"], case["tokens"], case["head_dim"], dtype)
        config = psa_b200.PSAConfig(block_n=case["block_n"], mask_ratios=RATIOS["mass"] if case["mode"] == "thresholdbound" else RATIOS[case["ratios"]],
                                    mask_mode=case["mode"])
        state["module"] = psa_b200.PSAAttention(config)
    elif kind == "preset":
        config = _preset(case)
        head_dim = MODELS[case["model"]][1]
        tokens, text = _preset_tokens(case), config.text_length
        cog = case["model"].startswith("CogVideo")
        q, k, v = _fields(seed, 1, case["heads"], tokens, head_dim, dtype, (config.depth, config.height, config.width), text)
        token_major = lambda x: x.transpose(1, 2).contiguous().transpose(1, 2)
        state["q"], state["k"], state["v"] = (q, k, token_major(v)) if cog else (token_major(q), token_major(k), token_major(v))
        state["rotary"] = _rotary(tokens, head_dim, text)
        state["module"] = PyramidSparseAttention(config, inference_num=50, layer_num=30, model_type="cogvideo" if cog else case["model"])
    elif kind == "train":
        q, k, v = _fields(seed, case["batch"], case["heads"], case["tokens"], case["head_dim"], dtype)
        state["q"], state["k"], state["v"] = (x.requires_grad_() for x in (q, k, v))
        state["mask"] = _random_level_mask(seed, case["batch"], case["heads"], case["tokens"])
        state["do"] = torch.randn(q.shape, device=DEVICE, dtype=dtype)
        state["fn"] = psa_b200.legacy_sparse_attention_factory(128, 32, 128, causal=True)
    else:
        q, k, v = _fields(seed, 1, case["heads"], case["tokens"], 128, dtype)
        if case["train"]:
            q, k, v = (x.requires_grad_() for x in (q, k, v))
            state["do"] = torch.randn(q.shape, device=DEVICE, dtype=dtype)
        state["q"], state["k"], state["v"] = q, k, v
        state["module"] = PyramidAdaptiveBlockSparseAttnTrain(CausalConfig(), layer_idx=0)
    return state


def run(state):
    q, k, v = state["q"], state["k"], state["v"]
    if state["kind"] == "module":
        return state["module"](q, k, v)
    if state["kind"] == "preset":
        with torch.no_grad():
            return state["module"](q, k, v, 0, rotary=state["rotary"])
    out = state["fn"](q, k, v, state["mask"]) if state["kind"] == "train" else state["module"](q, k, v)
    if "do" not in state:
        return out
    return [out.detach(), *torch.autograd.grad(out, (q, k, v), state["do"])]


# ------------------------------------------------------------------------------------------------ work and tolerance
def _rank_density(ratios):
    return sum((end - start) / level for level, (start, end) in ratios.items() if level)


def work(case):
    """q, k, v read once and the output written once (gradients: the upstream one read, three written).  Operations: the
    two products over the keys that survive (five more in a backward pass) and the product of the sampled quarters of q
    and k that the block scores are made of (causal site: groups of 16 tokens, half of the square)."""
    size = 4 if case["dtype"] == "f32" else 2
    causal = case["kind"] in ("train", "causal")
    backward = case["kind"] == "train" or case.get("train", False)
    if case["kind"] == "preset":
        config = _preset(case)
        batch, heads, tokens, head_dim = 1, case["heads"], _preset_tokens(case), MODELS[case["model"]][1]
        density = MASS_DENSITY[case["model"]] if config.mask_mode == "thresholdbound" else _rank_density(config.mask_ratios)
    elif case["kind"] == "causal":
        batch, heads, tokens, head_dim, density = 1, case["heads"], case["tokens"], 128, CAUSAL_DENSITY
    else:
        batch, heads, tokens, head_dim = case["batch"], case["heads"], case["tokens"], case["head_dim"]
        density = 0.46 if case["kind"] == "train" else MASS_DENSITY["module"] if case["mode"] == "thresholdbound" else _rank_density(RATIOS[case["ratios"]])
    square = float(batch * heads) * tokens * tokens * head_dim * (0.5 if causal else 1.0)
    estimate = 0.0 if case["kind"] == "train" else 2.0 * square / 16.0
    return {"bytes": batch * heads * tokens * head_dim * size * (8 if backward else 4),
            "flops": 4.0 * square * density * (3.5 if backward else 1.0) + estimate}


def tolerance(case):
    """About four times what two correct implementations at one precision show (tensor-core kernels against the scalar
    ones, 1560 to 75600 tokens): bf16 2.4e-3 (gradients 2.1e-3), f16 3e-4, or 4e-3 where a score that lands on the other
    side of a rounding boundary moves a block across a rank boundary; then a single value is off by up to a fifth (bf16)
    or a third (f16) of the result's size.  fp32 differs by its order of summation only."""
    if case["dtype"] == "f32":
        return {"rel": 1e-5}
    return {"rel": 1e-2, "max": 0.7}
