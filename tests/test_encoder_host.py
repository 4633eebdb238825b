"""What the host side of the whole-encoder calls refuses or leaves to the layer-by-layer forms, on the CPU: nothing is launched.

The native encoder is made over CPU tensors here, whose addresses only the library's geometry checks see; its `launch` is
replaced where a test reaches it.
"""

from __future__ import annotations

import pytest
import torch

from fastforks_b200 import _lib, encoder
from fastforks_b200.flash64 import Flash64
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
    """A ViT on the CPU that would take its native form where the arguments allow it; a launch fails the test."""
    enc = ViTEncoder(CFG, seeded_state(CFG), device="cpu", dtype=torch.float16)
    enc.scales = {k: v.float() for k, v in enc.scales.items()}
    native = enc._make_native()  # noqa: SLF001
    monkeypatch.setattr(native, "launch", lambda *a, **k: pytest.fail("launched"))
    monkeypatch.setattr(enc, "_native_now", lambda: native)
    monkeypatch.setattr(Flash64, "_run", staticmethod(lambda variant, q, k, v, scale: v.contiguous()))
    return enc


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
    with pytest.raises(KeyError):
        vit.intermediate(torch.zeros(1, 3, 28, 28), (0, 2))
