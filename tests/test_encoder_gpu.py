"""The encoder's own kernels at the sizes where they can go wrong, through the whole-encoder call, against float32 torch.

Layer norms alone are an encoder without blocks and one tap; windows, gated hidden layers, patches and the neck are one
block (or none) with seeded parameters. The norms' tolerance is that of one rounding to the output's type and of float32
sums (2^-11 or 2^-8 of the value, and 2^-16 for the sums' own error at unit scale); the others take the repository's
relative bar (`assert_close`), whose 2e-2 of the peak covers the eight or so fp16 roundings of a block many times over.
"""

from __future__ import annotations

import pytest
import torch
import torch.nn.functional as F  # noqa: N812

import fastforks_b200 as ff
from conftest import assert_close
from fastforks_b200 import encoder
from fastforks_b200.sam import SamConfig, SamEncoder, sam_state_shapes
from fastforks_b200.vit import ViTConfig, ViTEncoder, state_shapes

pytestmark = pytest.mark.gpu


def params(names: dict[str, tuple[int, ...]], seed: int) -> dict[str, torch.Tensor]:
    gen = torch.Generator().manual_seed(seed)
    return {k: (torch.randn(*s, generator=gen) / (s[-1] ** 0.5 if len(s) > 1 else 2.0) + (1.0 if k.endswith("norm_w") else 0.0)).half().cuda() for k, s in names.items()}


@pytest.mark.parametrize("dim", [64, 192, 256, 320, 576, 768, 1024, 1216, 1536, 1728, 2048])
@pytest.mark.parametrize("rows", [1, 5, 1203])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_layer_norm_at_every_row_length(dim: int, rows: int, dtype: torch.dtype) -> None:
    gen = torch.Generator().manual_seed(dim + rows)
    x = (torch.randn(rows, dim, generator=gen) * 3 + 1).to(dtype).cuda()
    w, b = (torch.randn(dim, generator=gen).to(dtype).cuda() for _ in range(2))
    enc = encoder.NativeEncoder([], dtype=dtype, dim=dim, heads=dim // 64, hidden=64, ffn=encoder.FFN_GELU, eps=1e-6)
    out = torch.full((rows + 1, dim), float("nan"), dtype=dtype, device="cuda")
    enc.launch(enc.describe(1, (1, rows), 0, 0, 0, {"x": 1, "norm_w": w.data_ptr(), "norm_b": b.data_ptr()}), x.device, x=x, taps=[(-1, out)])
    ref = F.layer_norm(x.double(), (dim,), w.double(), b.double(), 1e-6)
    assert ((out[:rows].double() - ref).abs() <= ref.abs() * 2.0 ** (-11 if dtype == torch.float16 else -8) + 2.0**-16).all()
    assert out[rows].isnan().all()  # the row behind the last one is not touched


def block_reference(x: torch.Tensor, p: dict[str, torch.Tensor], heads: int, window: int, ffn: int) -> torch.Tensor:
    """One block on `[B, gh, gw, C]`, float32."""
    p = {k: v.float() for k, v in p.items()}
    b, gh, gw, c = x.shape
    y = F.layer_norm(x, (c,), p["norm1_w"], p["norm1_b"], 1e-5)
    ws = window or 1
    ph, pw = -gh % ws, -gw % ws
    hp, wp = gh + ph, gw + pw
    y = F.pad(y, (0, 0, 0, pw, 0, ph))
    y = y.view(b, hp // ws, ws, wp // ws, ws, c).permute(0, 1, 3, 2, 4, 5).reshape(-1, ws * ws, c) if window else y.reshape(b, gh * gw, c)
    q, k, v = F.linear(y, p["qkv_w"], p["qkv_b"]).view(*y.shape[:2], 3, heads, 64).permute(2, 0, 3, 1, 4)
    y = F.linear(((q @ k.transpose(-1, -2) * 0.125).softmax(-1) @ v).transpose(1, 2).reshape(y.shape), p["proj_w"], p["proj_b"])
    if window:
        y = y.view(b, hp // ws, wp // ws, ws, ws, c).permute(0, 1, 3, 2, 4, 5).reshape(b, hp, wp, c)[:, :gh, :gw]
    x = x + y.reshape(x.shape)
    y = F.linear(F.layer_norm(x, (c,), p["norm2_w"], p["norm2_b"], 1e-5), p["fc1_w"], p["fc1_b"])
    if ffn == encoder.FFN_SWIGLU:
        gate, up = y.chunk(2, -1)
        y = F.silu(gate) * up
    else:
        y = F.gelu(y, approximate="none" if ffn == encoder.FFN_GELU else "tanh")
    return x + F.linear(y, p["fc2_w"], p["fc2_b"])


@pytest.mark.parametrize(("b", "grid", "window", "heads", "hidden", "ffn"), [
    (1, (1, 1), 2, 1, 8, encoder.FFN_GELU),  # one token in a window of four
    (2, (5, 9), 4, 2, 104, encoder.FFN_GELU),  # windows padded below and to the right
    (1, (28, 14), 14, 3, 256, encoder.FFN_GELU_TANH),  # no padding
    (3, (13, 30), 14, 1, 72, encoder.FFN_GELU),
    (1, (3, 5), 0, 1, 344, encoder.FFN_SWIGLU),  # gated hidden layers whose last column tile is ragged
    (2, (11, 13), 0, 5, 136, encoder.FFN_SWIGLU),
    (1, (20, 20), 0, 2, 8, encoder.FFN_SWIGLU),
])  # fmt: skip
def test_one_block_of_every_kind(b: int, grid: tuple[int, int], window: int, heads: int, hidden: int, ffn: int) -> None:
    c = heads * 64
    wide = 2 * hidden if ffn == encoder.FFN_SWIGLU else hidden
    p = params({"norm1_w": (c,), "norm1_b": (c,), "qkv_w": (3 * c, c), "qkv_b": (3 * c,), "proj_w": (c, c), "proj_b": (c,), "norm2_w": (c,),
                "norm2_b": (c,), "fc1_w": (wide, c), "fc1_b": (wide,), "fc2_w": (c, hidden), "fc2_b": (c,)}, seed=hidden)  # fmt: skip
    enc = encoder.NativeEncoder([p | {"window": window}], dtype=torch.float16, dim=c, heads=heads, hidden=hidden, ffn=ffn, eps=1e-5)
    x = torch.randn(b, *grid, c, generator=torch.Generator().manual_seed(c)).half().cuda()
    ref = block_reference(x.float(), p, heads, window, ffn)
    enc.launch(enc.describe(b, grid, 0, 0, 1, {"x": 1}), x.device, x=x)
    assert ff.device_status() == 0
    assert_close(x.float().cpu().numpy(), ref.cpu().numpy(), unit_scale=False, what=f"{b} {grid} {window} {hidden}")


@pytest.mark.parametrize(("b", "grid", "window", "hidden", "ffn"), [(7, (39, 40), 0, 768, encoder.FFN_GELU), (7, (7, 223), 0, 776, encoder.FFN_SWIGLU), (7, (40, 40), 14, 1536, encoder.FFN_GELU_TANH), (9, (40, 40), 0, 768, encoder.FFN_GELU), (9, (40, 41), 0, 776, encoder.FFN_SWIGLU), (9, (40, 41), 14, 1536, encoder.FFN_GELU_TANH)])  # fmt: skip
def test_one_block_on_either_side_of_going_backwards(b: int, grid: tuple[int, int], window: int, hidden: int, ffn: int) -> None:
    """A qkv tensor of the tokens just below and just above 48 MiB, from which on some products take the rows from the last to the first, the
    same with padded windows, and larger ones."""
    test_one_block_of_every_kind(b, grid, window, 12, hidden, ffn)


@pytest.mark.parametrize(("b", "grid", "patch", "extra", "prefix", "channels"), [
    (1, (1, 1), 2, (0, 0), 0, 8),
    (2, (3, 5), 14, (0, 0), 1, 0),  # 588 pixels of a patch in rows of 592
    (1, (7, 4), 16, (10, 6), 0, 256),  # pixels behind the last whole patch
    (3, (9, 33), 10, (2, 0), 0, 136),
])  # fmt: skip
@pytest.mark.parametrize("image_dtype", [torch.float32, torch.float16])
def test_patches_and_neck(b: int, grid: tuple[int, int], patch: int, extra: tuple[int, int], prefix: int, channels: int, image_dtype: torch.dtype) -> None:
    """An encoder without blocks: patch embedding, then (tokens, final norm) or (tokens, neck)."""
    c, (gh, gw) = 128, grid
    k = 3 * patch * patch
    p = params({"patch_w": (c, k), "start": (prefix + gh * gw, c), "norm_w": (c,), "norm_b": (c,)}, seed=patch)
    images = torch.randn(b, 3, gh * patch + extra[0], gw * patch + extra[1], generator=torch.Generator().manual_seed(k)).half().to(image_dtype).cuda()
    tokens = F.conv2d(images.float(), p["patch_w"].float().view(c, 3, patch, patch), stride=patch)[:, :, :gh, :gw].flatten(2).transpose(1, 2)
    tokens = F.pad(tokens, (0, 0, prefix, 0)) + p["start"].float()
    padded = F.pad(p["patch_w"], (0, -k % 8)).contiguous()
    enc = encoder.NativeEncoder([], dtype=torch.float16, dim=c, heads=2, hidden=64, ffn=encoder.FFN_GELU, eps=1e-6)
    fields = {"images": 1, "image_dtype": encoder._lib.F32 if image_dtype == torch.float32 else encoder._lib.F16, "height": images.shape[2],  # noqa: SLF001
              "width": images.shape[3], "patch": patch, "patch_w": padded.data_ptr(), "patch_k": padded.shape[1], "start": p["start"].data_ptr()}  # fmt: skip
    if channels == 0:
        out = torch.empty(b, prefix + gh * gw, c, dtype=torch.float16, device="cuda")
        fields |= {"norm_w": p["norm_w"].data_ptr(), "norm_b": p["norm_b"].data_ptr()}
        enc.launch(enc.describe(b, grid, prefix, 0, 0, fields), images.device, images=images, taps=[(-1, out)])
        ref = F.layer_norm(tokens, (c,), p["norm_w"].float(), p["norm_b"].float(), 1e-6)
    else:
        n = params({"w0": (channels, c), "n0_w": (channels,), "n0_b": (channels,), "w1": (channels, 9 * channels), "n1_w": (channels,), "n1_b": (channels,)}, seed=channels)
        out = torch.empty(b, channels, gh, gw, dtype=torch.float16, device="cuda")
        fields |= {f"neck_{name}": t.data_ptr() for name, t in n.items()} | {"neck_out": 1, "neck_channels": channels, "neck_eps": 1e-6}
        enc.launch(enc.describe(b, grid, prefix, 0, 0, fields), images.device, images=images, neck_out=out)
        n = {name: t.float() for name, t in n.items()}
        y = F.layer_norm(F.linear(tokens, n["w0"]), (channels,), n["n0_w"], n["n0_b"], 1e-6).transpose(1, 2).view(b, channels, gh, gw)
        y = F.conv2d(y, n["w1"].view(channels, 3, 3, channels).permute(0, 3, 1, 2), padding=1)
        ref = F.layer_norm(y.permute(0, 2, 3, 1), (channels,), n["n1_w"], n["n1_b"], 1e-6).permute(0, 3, 1, 2)
    assert ff.device_status() == 0
    assert_close(out.float().cpu().numpy(), ref.cpu().numpy(), unit_scale=False, what=f"{b} {grid} {patch} {channels}")


def random_state(shapes: dict[str, tuple[int, ...]], seed: int) -> dict[str, torch.Tensor]:
    """Every parameter different from those of another seed, but `pos_embed`, which an encoder may read once."""
    gen = torch.Generator().manual_seed(seed)
    state = {k: torch.randn(*s, generator=gen) * (0.1 if len(s) > 1 else 0.3) + (1.0 if "norm" in k and k.endswith("weight") else 0.0) for k, s in shapes.items()}
    state["pos_embed"] = torch.randn(*shapes["pos_embed"], generator=torch.Generator().manual_seed(0))
    return state


def give(held: dict[str, torch.Tensor], values: dict[str, torch.Tensor], how: str) -> None:
    for name, value in values.items():
        if how == "in place":
            held[name].copy_(value)
        elif how == "entry":
            held[name] = value.clone()
        else:
            held[name].data = value.clone()


@pytest.mark.parametrize("how", ["in place", "entry", "storage"])
@pytest.mark.parametrize(("patch", "ffn", "layerscale"), [(14, "mlp", True), (16, "swiglu", False)])
def test_vit_forward_follows_its_parameters(how: str, patch: int, ffn: str, layerscale: bool) -> None:  # noqa: FBT001
    """An encoder whose parameters were written in place, replaced in its dictionaries or given other storage computes what a
    new encoder of those parameters does."""
    cfg = ViTConfig(128, 2, 2, patch, 4 * patch, ffn=ffn, layerscale=layerscale)
    enc = ViTEncoder(cfg, random_state(state_shapes(cfg), 1), device="cuda")
    images = torch.rand(2, 3, 3 * patch, 5 * patch, generator=torch.Generator().manual_seed(3)).cuda()
    before = enc(images)
    other = ViTEncoder(cfg, random_state(state_shapes(cfg), 2), device="cuda")
    give(enc.w, other.w, how)
    give(enc.scales, other.scales, how)
    with torch.no_grad():
        x = torch.randn(1, 9, 128, generator=torch.Generator().manual_seed(4)).half().cuda()
        assert torch.equal(enc.block(1, x.clone()), other.block(1, x.clone()))
    after, want = enc(images), other(images)
    assert torch.equal(after, want) and not torch.equal(after, before)
    assert all(torch.equal(a, b) for a, b in zip(enc.intermediate(images, (0, 1)), other.intermediate(images, (0, 1)), strict=True))
    assert ff.device_status() == 0


@pytest.mark.parametrize("how", ["in place", "entry", "storage"])
@pytest.mark.parametrize("patch", [14, 16])
def test_sam_forward_follows_its_parameters(how: str, patch: int) -> None:
    cfg = SamConfig(img=6 * patch, patch=patch, dim=128, depth=2, heads=2, out_chans=24, window=4, global_blocks=(1,))
    enc = SamEncoder(cfg, random_state(sam_state_shapes(cfg), 1), device="cuda")
    images = torch.rand(2, 3, cfg.img, cfg.img, generator=torch.Generator().manual_seed(3)).cuda()
    before = enc(images)
    state = random_state(sam_state_shapes(cfg), 2)
    state["pos_embed"] = state["pos_embed"] + 1.0
    other = SamEncoder(cfg, state, device="cuda")
    give(enc.w, other.w, how)
    after, want = enc(images), other(images)
    assert torch.equal(after, want) and not torch.equal(after, before)
    assert ff.device_status() == 0


def test_the_neck_alone_waits_for_its_weights() -> None:
    """Given tokens, no blocks: the neck's first product is the first kernel of the call, right behind the one that writes its
    weights and tokens."""
    c, channels, grid = 768, 256, (64, 64)
    weights = params({"w0": (channels, c), "n0_w": (channels,), "n0_b": (channels,), "w1": (channels, 9 * channels), "n1_w": (channels,), "n1_b": (channels,)}, seed=1)
    tokens = torch.randn(1, 64 * 64, c, generator=torch.Generator().manual_seed(2)).half().cuda()
    enc = encoder.NativeEncoder([], dtype=torch.float16, dim=c, heads=12, hidden=64, ffn=encoder.FFN_GELU, eps=1e-6)
    held, x = {k: torch.zeros_like(t) for k, t in weights.items()}, torch.zeros_like(tokens)
    fields = {f"neck_{name}": t.data_ptr() for name, t in held.items()} | {"x": 1, "neck_out": 1, "neck_channels": channels, "neck_eps": 1e-6}
    described = enc.describe(1, grid, 0, 0, 0, fields)
    outs = [torch.empty(1, channels, *grid, dtype=torch.float16, device="cuda") for _ in range(3)]
    enc.launch(described, x.device, x=x, neck_out=outs[0])
    for out in outs[1:]:
        x.copy_(tokens)
        for name, t in held.items():
            t.copy_(weights[name]) if name != "w0" else None
        held["w0"].copy_(weights["w0"])  # last
        enc.launch(described, x.device, x=x, neck_out=out)
    torch.cuda.synchronize()
    assert torch.equal(outs[1], outs[2]) and not torch.equal(outs[0], outs[1])
    assert ff.device_status() == 0
