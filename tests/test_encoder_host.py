"""What the host side of the whole-encoder calls refuses or leaves to the layer-by-layer forms, on the CPU: nothing is launched.

The native encoder is made over CPU tensors here, whose addresses only the library's geometry checks see; its `launch` is
replaced where a test reaches it.
"""

from __future__ import annotations

import copy
import pickle

import pytest
import torch

from fastforks_b200 import _lib, encoder
from fastforks_b200.flash64 import Flash64, is_stock
from fastforks_b200.sam import SamConfig, SamEncoder, sam_seeded_state
from fastforks_b200.vit import ViTConfig, ViTEncoder, seeded_state


@pytest.fixture(scope="module", autouse=True)
def _library() -> None:
    if _lib.needs_build():
        _lib.build()
    _lib.library.cache_clear()
    _lib.library()


CFG = ViTConfig(128, 2, 2, 14, 56)


@pytest.fixture
def vit(monkeypatch: pytest.MonkeyPatch) -> ViTEncoder:
    """A ViT on the CPU that takes its native form where the arguments allow it; `launched` lists the launches, which do nothing."""
    enc = ViTEncoder(CFG, seeded_state(CFG), device="cpu", dtype=torch.float16)
    enc.scales = {k: v.float() for k, v in enc.scales.items()}
    native = enc._make_native()  # noqa: SLF001
    enc.launched = []
    monkeypatch.setattr(native, "launch", lambda described, *a, **k: enc.launched.append(described[0].n_blocks))
    monkeypatch.setattr(enc, "_native_now", lambda: native)
    return enc


GEOMETRY = {"dtype": torch.float16, "dim": 128, "heads": 2, "hidden": 72, "ffn": encoder.FFN_SWIGLU, "eps": 1e-6}
SHAPES = {"norm1_w": (128,), "norm1_b": (128,), "qkv_w": (384, 128), "qkv_b": (384,), "proj_w": (128, 128), "proj_b": (128,), "gamma1": (128,),
          "norm2_w": (128,), "norm2_b": (128,), "fc1_w": (144, 128), "fc1_b": (144,), "fc2_w": (128, 72), "fc2_b": (128,), "gamma2": (128,),
          "rel_pos_h": (7, 64), "rel_pos_w": (7, 64)}  # fmt: skip


def block(window: int = 4) -> dict:
    return {k: torch.zeros(*s, dtype=torch.float32 if k.startswith("gamma") else torch.float16) for k, s in SHAPES.items()} | {"window": window}


@pytest.mark.parametrize(("first", "count"), [(0, 3), (2, 1), (-1, 1), (-1, 2), (1, 2), (3, 0), (0, -1)])
def test_blocks_that_do_not_exist_are_refused(vit: ViTEncoder, first: int, count: int) -> None:
    native = vit._native_now()  # noqa: SLF001
    native.describe(1, (4, 1), 0, 0, 2, {"x": 1})
    native.describe(1, (4, 1), 0, 2, 0, {"x": 1})
    with pytest.raises(ValueError, match="of 2"):
        native.describe(1, (4, 1), 0, first, count, {"x": 1})


@pytest.mark.parametrize("i", [2, -1, 7, True])
def test_block_numbers_out_of_range_raise_as_the_layers_do(vit: ViTEncoder, i: int) -> None:
    with pytest.raises(KeyError):
        vit.block(i, torch.zeros(1, 5, 128, dtype=torch.float16))
    assert vit.launched == []
    with pytest.raises(KeyError):
        vit.intermediate(torch.zeros(1, 3, 28, 28), (0, 2))
    assert vit.launched == [1, 1]  # the blocks that do exist, one by one
    vit.block(1, torch.zeros(1, 5, 128, dtype=torch.float16))
    vit.intermediate(torch.zeros(1, 3, 28, 28), (0, 1))
    assert vit.launched == [1, 1, 1, 2]


@pytest.mark.parametrize("width", [64, 120, 192, 1])
def test_tokens_of_another_width_are_left_to_the_layers(vit: ViTEncoder, width: int) -> None:
    with pytest.raises(RuntimeError, match="normalized_shape"):
        vit.block(0, torch.zeros(1, 5, width, dtype=torch.float16))
    assert vit.launched == []


def test_tensors_on_another_device_are_refused(vit: ViTEncoder) -> None:
    with pytest.raises(RuntimeError):  # torch's device mismatch
        vit.block(0, torch.zeros(1, 5, 128, dtype=torch.float16, device="meta"))
    assert vit._forward_native(torch.zeros(1, 3, 28, 28, device="meta"), 2, (1,)) is None  # noqa: SLF001
    native = encoder.NativeEncoder([block()], **GEOMETRY)
    described = native.describe(1, (4, 1), 0, 0, 0, {"x": 1})
    meta = torch.zeros(4, 128, dtype=torch.float16, device="meta")
    with pytest.raises(ValueError, match="parameters on cpu"):
        native.launch(described, meta.device, x=meta)
    with pytest.raises(ValueError, match="launch on cpu"):
        native.launch(described, torch.device("cpu"), x=meta)


@pytest.mark.parametrize("name", SHAPES)
def test_parameters_the_kernels_would_read_past_are_refused(name: str) -> None:
    """Shape, type, device, layout and alignment of every parameter whose address goes into the table."""
    good = block()
    encoder.NativeEncoder([good], **GEOMETRY)
    t = good[name]
    shifted = torch.zeros(t.numel() + 4, dtype=t.dtype)[2:][: t.numel()].view_as(t)  # 4 or 8 bytes off
    wrong = [t[:-1].clone(), t.expand(2, *t.shape).contiguous(), t.double(), t.to("meta"), shifted]
    if t.dim() == 2:  # noqa: PLR2004
        wrong += [t.T.contiguous().T, t[:, :-8].clone()]
    for bad in wrong:
        with pytest.raises(ValueError, match=name):
            encoder.NativeEncoder([good, good | {name: bad}], **GEOMETRY)
    if not name.startswith(("gamma", "rel_pos")):
        with pytest.raises(ValueError, match=name):
            encoder.NativeEncoder([{k: v for k, v in good.items() if k != name}], **GEOMETRY)


def test_relative_tables_of_a_grid_are_compared_with_it() -> None:
    native = encoder.NativeEncoder([block(0)], **GEOMETRY)
    native.describe(1, (4, 4), 0, 0, 1, {"x": 1})
    for grid in ((5, 5), (2, 2), (4, 2), (4, 5)):
        with pytest.raises(ValueError, match="does not fit"):
            native.describe(1, grid, 0, 0, 1, {"x": 1})


@pytest.mark.parametrize("name", ["blocks.0.norm1.weight", "blocks.1.attn.qkv.weight", "blocks.1.mlp.fc2.bias", "blocks.0.ls1.gamma"])
def test_a_state_of_other_shapes_is_left_to_the_layers(name: str) -> None:
    state = seeded_state(CFG)
    state[name] = state[name][:-8].clone()
    enc = ViTEncoder(CFG, state, device="cpu", dtype=torch.float16)
    assert enc._make_native() is None  # noqa: SLF001


VIT_OTHERS = ("cls_token", "patch_embed.proj.weight", "patch_embed.proj.bias", "norm.weight", "norm.bias")
SAM_OTHERS = ("pos_embed", "patch_embed.proj.weight", "patch_embed.proj.bias", "neck.0.weight", "neck.1.weight", "neck.1.bias", "neck.2.weight", "neck.3.weight", "neck.3.bias")


@pytest.mark.parametrize("name", [*(f"vit {n}" for n in VIT_OTHERS), *(f"sam {n}" for n in SAM_OTHERS)])
def test_parameters_beside_the_blocks_are_looked_at_too(name: str) -> None:
    """Slices of a flat buffer that begin off a 16-byte boundary, strided views and other shapes run layer by layer."""
    kind, name = name.split()
    if kind == "vit":
        enc = ViTEncoder(CFG, seeded_state(CFG), device="cpu", dtype=torch.float16)
        enc.scales = {k: v.float() for k, v in enc.scales.items()}
    else:
        cfg = SamConfig(img=96, patch=16, dim=128, depth=2, heads=2, out_chans=24, window=4, global_blocks=(1,))
        enc = SamEncoder(cfg, sam_seeded_state(cfg), device="cpu", dtype=torch.float16)
    assert enc._make_native() is not None  # noqa: SLF001
    t = enc.w[name]
    shifted = torch.zeros(t.numel() + 8, dtype=t.dtype)[2:][: t.numel()].view_as(t)
    for bad in (shifted, torch.zeros(*t.shape, 2, dtype=t.dtype)[..., 0], t[..., :-1].clone() if t.shape[-1] > 1 else t[:-1].clone()):
        enc.w[name] = bad
        assert enc._make_native() is None  # noqa: SLF001


def test_a_position_table_of_another_width_is_left_to_the_layers(vit: ViTEncoder) -> None:
    vit.pos_table = vit.pos_table[..., :64].contiguous()
    assert vit._forward_native(torch.zeros(1, 3, 28, 28), 2, (1,)) is None  # noqa: SLF001
    assert vit.launched == []


def test_patches_of_an_odd_side_are_left_to_the_layers(monkeypatch: pytest.MonkeyPatch) -> None:
    cfg = ViTConfig(128, 1, 2, 7, 28)
    enc = ViTEncoder(cfg, seeded_state(cfg), device="cpu", dtype=torch.float16)
    enc.scales = {k: v.float() for k, v in enc.scales.items()}
    native = enc._make_native()  # noqa: SLF001
    monkeypatch.setattr(enc, "_native_now", lambda: native)
    assert enc._forward_native(torch.zeros(1, 3, 28, 28), 1, (0,)) is None  # noqa: SLF001


def test_more_tokens_than_a_launch_holds_are_left_to_the_layers(vit: ViTEncoder) -> None:
    native = vit._native_now()  # noqa: SLF001
    assert native.try_describe(1 << 16, (1 << 12, 1), 0, 0, 1, {"x": 1}) is None
    assert native.try_describe(1 << 8, (1 << 12, 1), 0, 0, 1, {"x": 1}) is not None


@pytest.mark.parametrize("name", ["tokens", "blocks.1.attn.qkv.weight", "blocks.0.norm1.bias", "scale"])
def test_a_block_that_is_asked_for_gradients_is_left_to_the_layers(vit: ViTEncoder, name: str, monkeypatch: pytest.MonkeyPatch) -> None:
    """Attention and gemm refuse operands that require a gradient; so must the block they stand in."""
    x = torch.zeros(1, 5, 128, dtype=torch.float16)
    {"tokens": x, "scale": vit.scales["blocks.1.ls1.gamma"]}.get(name, vit.w.get(name)).requires_grad_()
    reached = []
    monkeypatch.setattr(ViTEncoder, "linear", lambda *a, **k: reached.append(a))
    with pytest.raises(AttributeError, match="view"):  # of what the replaced layer returned
        vit.block(1, x)
    assert reached and vit.launched == []
    with torch.no_grad():
        vit.block(1, x)
    assert vit.launched == [1]


def test_replaced_steps_are_seen(monkeypatch: pytest.MonkeyPatch) -> None:
    """A launcher or a step of the forward that a caller put in a model is what runs."""

    class Sub(ViTEncoder):
        def block(self, i: int, x: torch.Tensor) -> torch.Tensor:
            return super().block(i, x)

    class Plain(ViTEncoder):
        def checked(self, images: torch.Tensor) -> torch.Tensor:
            return images

    steps = ("tokens", "pos_embed", "linear", "block")
    enc = ViTEncoder(CFG, seeded_state(CFG), device="cpu")
    assert is_stock(enc.attn) and not encoder.overrides(enc, ViTEncoder, steps)
    assert encoder.overrides(Sub(CFG, seeded_state(CFG), device="cpu"), ViTEncoder, steps)
    assert not encoder.overrides(Plain(CFG, seeded_state(CFG), device="cpu"), ViTEncoder, steps)
    enc.block = lambda i, x: x
    assert encoder.overrides(enc, ViTEncoder, steps)
    assert not is_stock(lambda q, k, v, scale: q)
    launcher = Flash64("fh")
    assert is_stock(launcher)
    launcher._run = Flash64._run  # noqa: SLF001
    assert not is_stock(launcher)
    monkeypatch.setattr(Flash64, "_run", staticmethod(lambda *a: None))
    assert not is_stock(enc.attn)


@pytest.mark.parametrize("kind", ["vit", "sam"])
@pytest.mark.parametrize("duplicate", [copy.deepcopy, lambda enc: pickle.loads(pickle.dumps(enc))])  # noqa: S301
def test_encoders_can_be_copied_and_pickled(kind: str, duplicate) -> None:  # noqa: ANN001
    """The native table holds addresses of the original's tensors: a copy makes its own."""
    if kind == "vit":
        enc = ViTEncoder(CFG, seeded_state(CFG), device="cpu", dtype=torch.float16)
        enc.scales = {k: v.float() for k, v in enc.scales.items()}
    else:
        cfg = SamConfig(img=96, patch=16, dim=128, depth=2, heads=2, out_chans=24, window=4, global_blocks=(1,))
        enc = SamEncoder(cfg, sam_seeded_state(cfg), device="cpu", dtype=torch.float16)
    enc._native, enc._snapshot = enc._make_native(), encoder.Snapshot(enc.w)  # noqa: SLF001
    other = duplicate(enc)
    assert other._native is None and other._snapshot is None and enc._native is not None  # noqa: SLF001
    assert all(torch.equal(other.w[k], v) and other.w[k] is not v for k, v in enc.w.items())
    assert other._make_native() is not None  # noqa: SLF001
