"""What the speed of this framework is measured on: calls of its public entry points as a video diffusion pipeline makes them.

A case names a call (`kind`) and its sizes:

    layer     one sparse attention layer of a denoising step, mask predicted from this step's query and key
              (`SparseAttentionWithMap`, mean-pooled producer; selector `lines` or `mass`)
    guided    the same for both guidance branches of a layer in one call (`SparseAttentionWithMapCFG`)
    stored    one sparse attention layer under the mask of an earlier step (`SparseAttentionWithMap`, exact producer)
    refresh   the step on which the exact producer renews its map, fit and mask (`SparseAttentionWithMap`)
    dense     a warm-up step: dense attention (`SparseAttentionWithMap(..., use_dense=True)`)
    map       dense attention with the exact sparsity map (`flash_attn_with_sparsity_map`)
    prologue  what a processor does between the projections and the layer (`ops.qkv_prologue`)

The models are the three video transformers that `moddit_b200.synth.WORKLOADS` describes; query, key and value are its
synthetic activations (positional locality, per-head mixture for wan), so masks have the density and the shape that the
mask predictor finds on local attention.  Forward only: the framework has no backward pass.
"""
import logging
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "mod-dit_b200"))

from MoD.mod.attn_mask import SparseAttentionWithMap, SparseAttentionWithMapCFG  # noqa: E402
from MoD.mod.state import create_adaptive_mask_state  # noqa: E402
from MoD.mod.triton_flash_sparsity import flash_attn_with_sparsity_map  # noqa: E402
from moddit_b200 import ops, synth  # noqa: E402

LOG = logging.getLogger("perf")
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
# local window / vertical stripes / temporal diagonals, cycling over the heads
MIXTURE = ((1.0, 1.0, 1.0), (0.5, 0.5, 0.5, 4.0), (0.2, 1.2, 1.2))
WARMUP = 2              # both warm-up steps of a state collect features
MASS = 0.4              # share of the attention mass that the `mass` selector keeps


def _case(kind, model, heads, head_dim, block, frames, height, width, text, *, dtype="bf16", top_k=0, predict_T=5,
          selector="lines", gain=2.0, pad=0, keep=1.0):
    """pad: text tokens at the end that the padding mask switches off; keep: share of the blocks that the mask keeps."""
    return dict(kind=kind, model=model, heads=heads, head_dim=head_dim, block=block, frames=frames, height=height,
                width=width, text=text, dtype=dtype, top_k=top_k, predict_T=predict_T, selector=selector, gain=gain,
                pad=pad, keep=keep)


def listed():
    named = {
        # the smallest layer that the repository configures (two heads of 64, block 64): launches and host time count
        "smallest layer": _case("layer", "wan", 2, 64, 64, 4, 32, 32, 0, top_k=20, keep=0.326),
        # a rank's share of heads on a short clip: still bound by latency, several hundred work items
        "short clip": _case("layer", "hunyuan", 4, 128, 128, 8, 32, 32, 256, top_k=30, keep=0.315),
        # a medium clip through the cumulative-mass selector, in float16
        "medium clip, mass": _case("layer", "hunyuan", 8, 128, 128, 8, 64, 64, 256, dtype="fp16", selector="mass",
                                   gain=1.1, top_k=80, keep=0.161),
        # the headline layer: 117 frames at 768 x 1280 and 256 text tokens
        "hunyuan layer": _case("layer", "hunyuan", 24, 128, 128, 30, 48, 80, 256, top_k=300, keep=0.152),
        # 69 frames at 768 x 1280, heads of different kinds
        "wan layer": _case("layer", "wan", 40, 128, 128, 18, 48, 80, 0, top_k=160, predict_T=10, keep=0.183),
        # 44,880 + 224 tokens, head dimension 64, block 64: neither region is a whole number of blocks
        "cogvideox layer": _case("layer", "cogvideox", 48, 64, 64, 11, 48, 85, 224, top_k=100, predict_T=10, keep=0.123),
        # both guidance branches of a short text-first clip in float16
        "guided pair": _case("guided", "cogvideox", 16, 64, 64, 4, 64, 64, 256, dtype="fp16", top_k=60, keep=0.333),
        # the steps between two refreshes of the exact producer, with padded text
        "stored mask": _case("stored", "hunyuan", 24, 128, 128, 10, 48, 80, 256, top_k=100, pad=147, keep=0.172),
        # the step on which the exact producer renews its mask
        "refresh": _case("refresh", "wan", 40, 128, 128, 9, 48, 80, 0, top_k=80, predict_T=5, keep=0.17),
        # a warm-up step at head dimension 64
        "dense step": _case("dense", "cogvideox", 48, 64, 64, 5, 48, 85, 224, dtype="fp16"),
        # the map interface alone at the size of its own benchmark
        "map": _case("map", "hunyuan", 24, 128, 128, 31, 8, 16, 128, dtype="fp16"),
        # normalisation, rotation and layout of the headline layer's projections
        "prologue": _case("prologue", "hunyuan", 24, 128, 128, 30, 48, 80, 256),
    }
    return [dict(case, name=name) for name, case in named.items()]


def draw(rng):
    """A case of the same ranges: any kind and model, 4,000 to 115,000 tokens, up to the cost of the largest listed one."""
    kind = rng.choice(["layer"] * 5 + ["guided", "stored", "stored", "refresh", "dense", "map", "prologue"])
    model = rng.choice(["hunyuan", "wan", "cogvideox"])
    if kind == "guided" and model == "hunyuan":
        model = "cogvideox"
    head_dim = 64 if model == "cogvideox" else 128
    block = 64 if model == "cogvideox" else 128
    if rng.random() < 0.15:
        head_dim, block = rng.choice([(64, 64), (64, 128), (128, 64), (128, 128)])
    whole = kind in ("stored", "refresh", "map")          # the exact producer takes whole blocks only
    tokens = math.exp(rng.uniform(math.log(4000), math.log(115000 if head_dim == 128 else 46000)))
    height, width = rng.choice([32, 40, 48, 56, 64]), rng.choice([32, 48, 64, 80])
    if whole:
        width = 16 * max(1, width // 16)
        text = 0 if model == "wan" else 128 * rng.randint(1, 2)
    else:
        height, width = height + rng.choice([0, 0, 1, -3]), width + rng.choice([0, 0, 5, -1])
        text = 0 if model == "wan" else rng.randint(40, 300)
    # clips of fewer than three frames have smaller frames
    while tokens < 3 * height * width and height > 16:
        height //= 2
    if whole:
        height = 8 * max(1, height // 8)
    frames = max(3, min(round(tokens / (height * width)), 1000 * block // (height * width)))
    video = frames * height * width
    blocks = video // block
    top_k = max(8, round(blocks * rng.uniform(0.12, 0.34)))
    selector = "mass" if kind == "layer" and rng.random() < 0.2 else "lines"
    keep = 0.16 if selector == "mass" else min(1.0, 0.45 * top_k / blocks + 0.5 / frames + 2.0 * text / video)
    if kind in ("dense", "map", "prologue"):
        keep = 1.0
    case = _case(kind, model, 1, head_dim, block, frames, height, width, text,
                 dtype=rng.choice(["bf16", "bf16", "fp16"]), top_k=top_k, predict_T=rng.choice([5, 10]), selector=selector,
                 gain=1.1 if selector == "mass" else 2.0,
                 pad=rng.randint(1, text - 1) if kind == "stored" and model == "hunyuan" else 0, keep=round(keep, 3))
    one = work(case)
    most = min(48, int(20e12 / max(one["flops"], 1.0)), int(3e9 / one["bytes"]))
    case["heads"] = max(1, min(most, rng.choice([2, 3, 5, 8, 12, 16, 24, 30, 40, 48])))
    return case


def _tokens(case):
    video = case["frames"] * case["height"] * case["width"]
    return video, video + case["text"]


def _qkv(case, seed, branch=0):
    return synth.make_qkv(heads=case["heads"], grid=(case["frames"], case["height"], case["width"]),
                          head_dim=case["head_dim"], text_tokens=case["text"], text_first=case["model"] == "cogvideox",
                          seed=2 * seed + branch, gain=case["gain"],
                          axis_mix=MIXTURE if case["model"] == "wan" and case["heads"] > 2 else None,
                          device="cuda", dtype=DTYPES[case["dtype"]])


def _state(case):
    video, n = _tokens(case)
    state = create_adaptive_mask_state(case["model"], case["heads"], video, case["text"], case["height"] * case["width"],
                                       case["frames"], warmup_steps=WARMUP, top_k=case["top_k"],
                                       predict_T=case["predict_T"], block_size=case["block"])
    if case["kind"] in ("layer", "guided"):
        state["score_producer"] = "pooled"
    if case["selector"] == "mass":
        state.update(selector="cumulative_mass", mass_threshold=MASS)
    return state


def _projections(case, seed):
    """Projections, norm weights and rotary tables as the model's processor has them."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    video, n = _tokens(case)
    H, D, dtype = case["heads"], case["head_dim"], DTYPES[case["dtype"]]
    proj = [torch.randn(1, n, H * D, device="cuda", generator=g, dtype=torch.float32).to(dtype) for _ in range(3)]
    width = H * D if case["model"] == "wan" else D
    weight = [(1.0 + 0.1 * torch.randn(width, device="cuda", generator=g)).to(dtype) for _ in range(4)]
    first = case["text"] if case["model"] == "cogvideox" else 0
    pos = torch.arange(video, device="cuda", dtype=torch.float32)[:, None]
    freq = 10000.0 ** (-torch.arange(D // 2, device="cuda", dtype=torch.float32) * 2 / D)
    ang = pos * freq
    form = "even_cos_odd_sin" if case["model"] == "wan" else "elementwise"
    cos, sin = (t.repeat_interleave(2, dim=1).contiguous() for t in (ang.cos(), ang.sin()))
    kw = dict(num_heads=H, rope_cos=cos, rope_sin=sin, rope_form=form, rope_range=(first, first + video),
              pool_block_size=case["block"], q_weight=weight[0], k_weight=weight[1],
              norm={"hunyuan": "rms_head", "wan": "rms_all_heads", "cogvideox": "layer"}[case["model"]])
    if case["model"] == "cogvideox":
        kw.update(q_bias=weight[2] - 1.0, k_bias=weight[3] - 1.0)
    return proj, kw


def prepare(case, seed):
    kind = case["kind"]
    if kind == "prologue":
        proj, kw = _projections(case, seed)
        return dict(case=case, proj=proj, kw=kw)
    if kind == "guided":
        # two branches: (2, H, S, D) tensors and a state dict per branch, one collecting step behind them
        q, k, v = (torch.cat(pair) for pair in zip(_qkv(case, seed), _qkv(case, seed, 1)))
        states = [_state(case), _state(case)]
        SparseAttentionWithMapCFG(q, k, v, states, LOG, current_step=0)
        return dict(case=case, qkv=(q, k, v), states=states)
    q, k, v = _qkv(case, seed)
    if kind == "map":
        return dict(case=case, qkv=(q, k, v))
    state, video, n = _state(case), *_tokens(case)
    padding = None
    if case["pad"]:
        row = torch.arange(n, device="cuda") < n - case["pad"]
        padding = row.unsqueeze(0).expand(n, n)
    # the layer's earlier steps: one collecting step (pooled producer) or both (exact producer)
    if kind != "dense":
        for step in range(1 if kind == "layer" else WARMUP):
            SparseAttentionWithMap(q, k, v, state, LOG, pre_defined_mask=padding, current_step=step)
    return dict(case=case, qkv=(q, k, v), state=state, padding=padding)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "prologue":
        out, pools = ops.qkv_prologue(*state["proj"], **state["kw"])
        return {"qkv": out, "means": pools}
    q, k, v = state["qkv"]
    if kind == "guided":
        out, info = SparseAttentionWithMapCFG(q, k, v, state["states"], LOG, current_step=WARMUP)
        return {"out": out, "mask": info["mask"], "features": dict(state["states"][1]["features_history"][-1])}
    if kind == "map":
        video, _ = _tokens(case)
        out, sparsity = flash_attn_with_sparsity_map(q, k, v, 1.5e-4, case["block"], case["model"], video, case["text"])
        return {"out": out, "map": sparsity}
    layer = state["state"]
    if kind == "dense":
        out, _ = SparseAttentionWithMap(q, k, v, layer, LOG, current_step=0, use_dense=True)
        return {"out": out}
    step = WARMUP + (case["predict_T"] - 1 if kind == "refresh" else 0)
    out, info = SparseAttentionWithMap(q, k, v, layer, LOG, pre_defined_mask=state["padding"], current_step=step)
    result = {"out": out, "mask": info["mask"]}
    if kind in ("layer", "refresh"):
        result["features"] = dict(layer["features_history"][-1])
    if kind == "refresh":
        result["map"] = layer["prev_full_maps"]
    return result


def work(case):
    """Each input and output once; products of the kept blocks, plus the exact map's where it is made."""
    video, n = _tokens(case)
    H, D, kind = case["heads"] * (2 if case["kind"] == "guided" else 1), case["head_dim"], case["kind"]
    blocks = (n + case["block"] - 1) // case["block"]
    tensor = 2.0 * H * n * D
    if kind == "prologue":
        return {"bytes": 6 * tensor + 8.0 * video * D + 8.0 * H * blocks * D, "flops": 0.0}
    flops = 4.0 * H * D * n * n * (case["keep"] if kind in ("layer", "guided", "stored") else 1.0)
    size = 4 * tensor
    if kind in ("refresh", "map"):
        flops += 2.0 * H * D * (video * video)
        size += 2.0 * H * (video // case["block"]) ** 2
    if kind in ("layer", "guided", "stored", "refresh"):
        size += 1.0 * H * blocks * blocks
    return {"bytes": size, "flops": flops}


def tolerance(case):
    """About four times what was measured: the attention against masked attention in float64 (relative error 2.2e-3,
    largest difference 1.6e-2 of the root mean square, from 16-bit probabilities and outputs); the prologue against
    float64 without its intermediate roundings (2.9e-3, 2.1e-2).  Masks are whole values and stay the same; only where
    they come from the exact map, whose counts move by one with the last bits of the log-sum-exp, may a line at the
    rank-`top_k` cut change places with a nearly tied one (one of 80 lines of one head is 1e-4 of the blocks)."""
    if case["kind"] == "prologue":
        return {"rel": 1e-2, "max": 8e-2}
    if case["kind"] in ("stored", "refresh"):
        return {"rel": 1e-2, "max": 0.3, "differ": 1e-3}
    return {"rel": 1e-2, "max": 8e-2}
