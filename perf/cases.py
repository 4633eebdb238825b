"""What this framework is timed on: its public entry points at the sizes of its own configurations, and a generator of
more cases of the same ranges.

Kinds of case:

* `attn`: `Flash64` on views of a packed qkv tensor, the call of every ViT block;
* `masked`: `scaled_dot_product_attention` with an additive 16-bit mask (windowed blocks, whose bias is made once per
  block with rows padded to a multiple of eight columns);
* `sam_attn`: SAM's attention step, the producer of the decomposed bias and the attention that takes it;
* `dinov3`: the attention half of a DINOv3 block behind its norm: qkv layer, rotary embedding, attention, projection
  with LayerScale and residual;
* `vit`: a whole ViT encoder forward (`ViTEncoder`), or the intermediate outputs a depth head takes;
* `sam`: a whole SAM image encoder forward (`SamEncoder`).

Everything is inference; weights and inputs are seeded random values of the scale a trained or freshly made network has.
"""

from __future__ import annotations

import dataclasses
import math

import torch

import fastforks_b200 as ff
from fastforks_b200.sam import SAM_VIT_B, SamEncoder, sam_state_shapes
from fastforks_b200.vit import CONFIGS, ViTEncoder, state_shapes

HEAD_DIM = 64
SCALE = HEAD_DIM**-0.5
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}
DINOV3_PREFIX = 5  # class token and four registers


def listed() -> list[dict]:
    return [
        # One block's attention of ViT-B/16 on one 224 px image: the smallest call, bound by launch latency and host work.
        {"name": "attn-1x197", "kind": "attn", "batch": 1, "heads": 12, "tokens": 197, "dtype": "fp16"},
        # The same block on a full batch of a classifier: many short sequences, bound by memory.
        {"name": "attn-256x197", "kind": "attn", "batch": 256, "heads": 12, "tokens": 197, "dtype": "fp16"},
        # DINOv2 ViT-S/14 features of eight 518 px images: a long, ragged sequence on a few heads.
        {"name": "attn-8x1370", "kind": "attn", "batch": 8, "heads": 6, "tokens": 1370, "dtype": "fp16"},
        # DINOv2 ViT-g/14 on a large batch: the largest attention call.
        {"name": "attn-32x1370", "kind": "attn", "batch": 32, "heads": 24, "tokens": 1370, "dtype": "bf16"},
        # A windowed block: 7 x 7 windows folded into the heads, each with its own relative-position bias.
        {"name": "masked-8x192x49", "kind": "masked", "batch": 8, "heads": 192, "tokens": 49, "dtype": "fp16"},
        # SAM ViT-B at 1024 px, a windowed block: 25 windows of 14 x 14.
        {"name": "sam-attn-25x14", "kind": "sam_attn", "batch": 25, "heads": 12, "side": 14, "dtype": "fp16"},
        # SAM ViT-B at 1024 px, a global block: the 64 x 64 grid.
        {"name": "sam-attn-1x64", "kind": "sam_attn", "batch": 1, "heads": 12, "side": 64, "dtype": "fp16"},
        # DINOv3 ViT-L/16 features of 512 px images: linear layers and rotary embedding around the attention.
        {"name": "dinov3-32x512px", "kind": "dinov3", "batch": 32, "heads": 16, "grid_h": 32, "grid_w": 32, "dtype": "fp16"},
        # ViT-B/16 on one 224 px image, the interactive classifier: some hundred short kernels.
        {"name": "vit-b16-1", "kind": "vit", "model": "vit-b16", "batch": 1, "height": 224, "width": 224, "layers": "", "dtype": "fp16"},
        # The encoder call of Depth-Anything-V2-L on four 518 px images: four intermediate outputs for the depth head.
        {"name": "vit-l14-4", "kind": "vit", "model": "dinov2-vitl14", "batch": 4, "height": 518, "width": 518, "layers": "4,11,17,23", "dtype": "bf16"},
        # DINOv2 ViT-g/14 (SwiGLU) on a chunk of sixteen images: the largest forward.
        {"name": "vit-g14-16", "kind": "vit", "model": "dinov2-vitg14", "batch": 16, "height": 518, "width": 518, "layers": "", "dtype": "bf16"},
        # SAM ViT-B image encoder on one 1024 px image, what a user waits for before the first prompt.
        {"name": "sam-vit-b-1", "kind": "sam", "batch": 1, "img": 1024, "dtype": "fp16"},
    ]


def _log_int(rng, low: int, high: int) -> int:
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng) -> dict:
    kind = rng.choice(["attn", "attn", "masked", "sam_attn", "dinov3", "vit", "vit", "sam"])
    dtype = rng.choice(["fp16", "bf16"])
    if kind == "attn":
        tokens, heads = _log_int(rng, 33, 4608), rng.choice([3, 6, 12, 16, 24])
        most = min(32 * 24 * 1370**2 / (heads * tokens**2), 256 * 12 * 197 / (heads * tokens) * 2)
        return {"kind": kind, "batch": _log_int(rng, 1, max(1, min(256, int(most)))), "heads": heads, "tokens": tokens, "dtype": dtype}
    if kind == "masked":
        tokens, heads = rng.choice([49, 64, 98, 144, 196, 200, 256, _log_int(rng, 33, 1370)]), _log_int(rng, 4, 256)
        heads = max(1, min(heads, int(64e6 / tokens**2)))
        most = min(4e8 / (heads * tokens**2), 8e5 / (heads * tokens))
        return {"kind": kind, "batch": _log_int(rng, 1, max(1, min(64, int(most)))), "heads": heads, "tokens": tokens, "dtype": dtype}
    if kind == "sam_attn":
        side, heads = 2 * _log_int(rng, 3, 32), rng.choice([12, 16])
        most = min(4 * 4096**2 / side**4, 100 * 196 / side**2)
        return {"kind": kind, "batch": _log_int(rng, 1, max(1, int(most))), "heads": heads, "side": side, "dtype": dtype}
    if kind == "dinov3":
        grid_h, grid_w = rng.randint(14, 48), rng.randint(14, 48)
        most = 32 * 1029 / (grid_h * grid_w + DINOV3_PREFIX)
        return {"kind": kind, "batch": _log_int(rng, 1, max(1, int(most))), "heads": rng.choice([6, 12, 16]), "grid_h": grid_h, "grid_w": grid_w, "dtype": dtype}
    if kind == "vit":
        model = rng.choice(["vit-b16", "dinov2-vits14", "dinov2-vitb14", "dinov2-vitl14", "dinov2-vitg14"])
        cfg = CONFIGS[model]
        grid_h, grid_w = rng.randint(12, 40), rng.randint(12, 40)
        most = min(32, 16 * 1370 / (grid_h * grid_w + 1))
        layers = rng.choice(["", f"{cfg.depth // 2},{cfg.depth - 1}"])
        return {"kind": kind, "model": model, "batch": _log_int(rng, 1, max(1, int(most))), "height": grid_h * cfg.patch, "width": grid_w * cfg.patch,
                "layers": layers, "dtype": dtype}  # fmt: skip
    return {"kind": "sam", "batch": rng.randint(1, 4), "img": rng.choice([512, 640, 768, 1024]), "dtype": dtype}


def _weights(shapes: dict[str, tuple[int, ...]], gen: torch.Generator) -> dict[str, torch.Tensor]:
    """A seeded fp32 state dict on the GPU: matrices ~ N(0, 0.02), relative-position tables ~ N(0, 0.1), norm weights and
    LayerScale factors around 1, biases around 0."""
    state = {}
    for name, shape in shapes.items():
        t = torch.randn(shape, generator=gen, device="cuda")
        if name.endswith(".gamma") or (name.endswith(".weight") and ("norm" in name or name in ("neck.1.weight", "neck.3.weight"))):
            state[name] = t.mul_(0.02).add_(1.0)
        else:
            state[name] = t.mul_(0.1 if "rel_pos" in name else 0.02)
    return state


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[case["dtype"]]

    def randn(*shape: int, std: float = 1.0) -> torch.Tensor:
        return torch.randn(shape, generator=gen, device="cuda").mul_(std).to(dtype)

    kind, batch = case["kind"], case["batch"]
    state = {"kind": kind}
    if kind == "attn":
        state["qkv"] = randn(batch, case["tokens"], 3, case["heads"], HEAD_DIM)
        state["flash"] = ff.Flash64()
    elif kind == "masked":
        state["q"], state["k"], state["v"] = (randn(batch, case["heads"], case["tokens"], HEAD_DIM) for _ in range(3))
        state["mask"] = ff.tile_layout(randn(1, case["heads"], case["tokens"], case["tokens"]))
    elif kind == "sam_attn":
        side = state["side"] = case["side"]
        state["qkv"] = randn(batch, side * side, 3, case["heads"], HEAD_DIM)
        state["pos_h"], state["pos_w"] = (randn(2 * side - 1, HEAD_DIM, std=0.1) for _ in range(2))
    elif kind == "dinov3":
        heads, dim = case["heads"], case["heads"] * HEAD_DIM
        tokens = case["grid_h"] * case["grid_w"] + DINOV3_PREFIX
        state["heads"] = heads
        state["normed"], state["x"] = randn(batch, tokens, dim), randn(batch, tokens, dim)
        state["w_qkv"], state["b_qkv"] = randn(3 * dim, dim, std=dim**-0.5), randn(3 * dim, std=0.02)
        state["w_proj"], state["b_proj"] = randn(dim, dim, std=dim**-0.5), randn(dim, std=0.02)
        state["gamma"] = torch.rand(dim, generator=gen, device="cuda")
        state["cs"] = ff.rope_table(case["grid_h"], case["grid_w"], device="cuda")
        state["flash"] = ff.Flash64()
    elif kind == "vit":
        cfg = CONFIGS[case["model"]]
        state["encoder"] = ViTEncoder(cfg, _weights(state_shapes(cfg), gen), dtype=dtype)
        state["images"] = torch.rand(batch, 3, case["height"], case["width"], generator=gen, device="cuda")
        state["layers"] = tuple(int(i) for i in case["layers"].split(",") if i)
    else:
        cfg = dataclasses.replace(SAM_VIT_B, img=case["img"])
        state["encoder"] = SamEncoder(cfg, _weights(sam_state_shapes(cfg), gen), dtype=dtype)
        state["images"] = torch.rand(batch, 3, case["img"], case["img"], generator=gen, device="cuda")
    return state


@torch.no_grad()
def run(state: dict):
    kind = state["kind"]
    if kind == "attn":
        q, k, v = state["qkv"].unbind(2)
        return state["flash"](q, k, v, SCALE)
    if kind == "masked":
        return ff.scaled_dot_product_attention(state["q"], state["k"], state["v"], attn_mask=state["mask"])
    if kind == "sam_attn":
        q, k, v = state["qkv"].unbind(2)
        rel = ff.sam_rel_terms(q, state["pos_h"], state["pos_w"], state["side"])
        return ff.attention(q, k, v, scale=SCALE, rel=rel, layout="bnhd")
    if kind == "dinov3":
        b, n, c = state["x"].shape
        qkv = ff.gemm(state["normed"], state["w_qkv"], state["b_qkv"]).view(b, n, 3, state["heads"], HEAD_DIM)
        q, k, v = ff.rope_qk_(qkv, state["cs"], q_scale=SCALE).unbind(2)
        attended = state["flash"](q, k, v, 1.0).view(b, n, c)
        return ff.gemm(attended, state["w_proj"], state["b_proj"], scale=state["gamma"], res=state["x"])
    if kind == "vit" and state["layers"]:
        return state["encoder"].intermediate(state["images"], state["layers"])
    return state["encoder"](state["images"])


def _encoder_work(batch: int, tokens: int, dim: int, hidden: int, depth: int, gate: int) -> float:
    """FLOPs of `depth` blocks: qkv, projection, MLP (`gate` = 2: a SwiGLU's doubled first layer) and attention."""
    linear = 2.0 * batch * tokens * dim * (4 * dim + (1 + gate) * hidden)
    return depth * (linear + 4.0 * batch * tokens * tokens * dim)


def work(case: dict) -> dict:
    kind, b = case["kind"], case["batch"]
    if kind in ("attn", "masked"):
        n, h = case["tokens"], case["heads"]
        mask = 2.0 * h * n * n if kind == "masked" else 0.0
        return {"bytes": 8.0 * b * h * n * HEAD_DIM + mask, "flops": 4.0 * b * h * n * n * HEAD_DIM}
    if kind == "sam_attn":
        n, h, side = case["side"] ** 2, case["heads"], case["side"]
        return {"bytes": 8.0 * b * h * n * HEAD_DIM + 2 * 2 * (2 * side - 1) * HEAD_DIM, "flops": 4.0 * b * h * n * n * HEAD_DIM + 4.0 * b * h * n * side * HEAD_DIM}
    if kind == "dinov3":
        n, dim = case["grid_h"] * case["grid_w"] + DINOV3_PREFIX, case["heads"] * HEAD_DIM
        bytes_ = 2.0 * (3 * b * n * dim + 4 * dim * dim) + 256.0 * case["grid_h"] * case["grid_w"]
        return {"bytes": bytes_, "flops": 8.0 * b * n * dim * dim + 4.0 * b * n * n * dim}
    if kind == "vit":
        cfg = CONFIGS[case["model"]]
        layers = [int(i) for i in case["layers"].split(",") if i]
        depth = max(layers) + 1 if layers else cfg.depth
        n, gate = cfg.tokens(case["height"], case["width"]), 2 if cfg.ffn == "swiglu" else 1
        weights = depth * cfg.dim * (4 * cfg.dim + (1 + gate) * cfg.hidden) + 3 * cfg.patch**2 * cfg.dim + n * cfg.dim
        bytes_ = 2.0 * weights + 12.0 * b * case["height"] * case["width"] + 2.0 * b * n * cfg.dim * max(1, len(layers))
        patches = 2.0 * b * (n - 1) * 3 * cfg.patch**2 * cfg.dim
        return {"bytes": bytes_, "flops": _encoder_work(b, n, cfg.dim, cfg.hidden, depth, gate) + patches}
    cfg = SAM_VIT_B
    grid = case["img"] // cfg.patch
    n, windows = grid * grid, (-(-grid // cfg.window)) ** 2
    glob, local = len(cfg.global_blocks), cfg.depth - len(cfg.global_blocks)
    flops = glob * (8.0 * b * n * cfg.dim**2 + 4.0 * b * n * n * cfg.dim + 4.0 * b * n * grid * cfg.dim)
    wn = cfg.window**2  # the tokens that pad a window take part in its attention; the linear layers do not need them
    flops += local * (8.0 * b * n * cfg.dim**2 + windows * (4.0 * b * wn * wn * cfg.dim + 4.0 * b * wn * cfg.window * cfg.dim))
    flops += cfg.depth * 16.0 * b * n * cfg.dim**2
    flops += 2.0 * b * n * (3 * cfg.patch**2 * cfg.dim + cfg.dim * cfg.out_chans + 9 * cfg.out_chans**2)
    weights = cfg.depth * 12 * cfg.dim**2 + 3 * cfg.patch**2 * cfg.dim + n * cfg.dim + cfg.out_chans * (cfg.dim + 9 * cfg.out_chans)
    return {"bytes": 2.0 * weights + 12.0 * b * case["img"] ** 2 + 2.0 * b * n * cfg.out_chans, "flops": flops}


def tolerance(case: dict) -> dict:
    """16-bit operands and results, 32-bit sums: one operator is off by a few roundings of its result and of the
    probabilities; an encoder rounds its residual stream in every block."""
    whole = case["kind"] in ("vit", "sam")
    if case["dtype"] == "fp16":
        return {"rel": 5e-3 if whole else 2e-3}
    return {"rel": 2e-2 if whole else 1e-2}
