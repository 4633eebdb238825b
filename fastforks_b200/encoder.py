"""Host side of the whole-encoder calls (include/b200_encoder.h): one native call per forward.

`NativeEncoder` keeps what a model's forwards share - the table of the blocks' parameter pointers and, per input
geometry, a filled-in argument description - and launches a forward with two allocations (outputs and one workspace)
from torch's caching allocator. Nothing here computes.
"""

from __future__ import annotations

import ctypes
import logging
from typing import TYPE_CHECKING

import torch

from . import _lib
from .attention import reserve_workspace

if TYPE_CHECKING:
    from collections.abc import Sequence

_LOG = logging.getLogger("fastforks_b200")
FFN_GELU_TANH, FFN_SWIGLU, FFN_GELU = 0, 1, 2
MAX_DIM = 2048  # a row of the layer norms lives in one warp's registers
_DTYPES = {torch.float16: _lib.F16, torch.bfloat16: _lib.BF16}
BLOCK_TENSORS = tuple(name for name, kind in _lib.B200EncoderBlock._fields_ if kind is ctypes.c_void_p)  # noqa: SLF001
_REQUIRED = {name for name in BLOCK_TENSORS if name[:5] not in ("gamma", "rel_p")}
_SPLIT_MIN_KEYS = 257  # shorter sequences never use the attention workspace


def supported(dtype: torch.dtype, dim: int, heads: int, hidden: int) -> bool:
    """Whether the native forward takes an encoder of this shape."""
    return dtype in _DTYPES and dim == heads * 64 and dim <= MAX_DIM and hidden % 8 == 0


class HoldsNative:
    """What a model that holds a native encoder is copied and pickled as: without it, since it is made of addresses. It is made
    again from the copy's own tensors."""

    def __getstate__(self) -> dict:
        return {**self.__dict__, "_native": None, "_snapshot": None}


def check_parameter(name: str, t: torch.Tensor, shape: tuple[int, ...], dtype: torch.dtype, device: torch.device) -> None:
    """Refuse a parameter the kernels cannot read through its address alone.

    Raises:
        ValueError: It has another shape, type or device, or is not contiguous and 16-byte aligned.
    """
    if tuple(t.shape) != shape or t.dtype != dtype or t.device != device or not t.is_contiguous() or t.data_ptr() % 16:
        msg = (f"encoder: parameter {name} must be contiguous, 16-byte aligned {dtype} {list(shape)} on {device}, "
               f"got {list(t.shape)} {t.dtype} {t.device} strides {t.stride()}")  # fmt: skip
        raise ValueError(msg)


def overrides(model: object, base: type, methods: tuple[str, ...]) -> bool:
    """Whether a subclass of a model or an attribute set on it replaces one of `methods`, which the native call would pass by."""
    return (type(model) is not base and any(getattr(type(model), m) is not getattr(base, m) for m in methods)) or not vars(model).keys().isdisjoint(methods)


class Snapshot:
    """The tensors of a model's dictionaries as they were when their addresses were taken: a tensor put in another's place, or
    given other storage, is seen by `changed`, which every forward asks. (Values written in place need no looking at: the
    kernels read the tensors themselves.) The tensors are kept alive, so that no address is used again while it is in the table."""

    def __init__(self, *dicts: dict[str, torch.Tensor]) -> None:
        _lib.use_fast()
        self._host = _lib.fast
        self._native = None if self._host is None else self._host.snapshot(dicts)
        self._kept = None if self._native is not None else self._facts(dicts)

    @staticmethod
    def _facts(dicts: tuple[dict[str, torch.Tensor], ...]) -> list[tuple]:
        return [(id(t), t.data_ptr(), t.shape, t.stride(), t) for d in dicts for t in d.values()]

    def changed(self, *dicts: dict[str, torch.Tensor]) -> bool:
        if self._native is not None:
            return not self._host.unchanged(self._native, dicts)
        return [f[:-1] for f in self._kept] != [f[:-1] for f in self._facts(dicts)]


class NativeEncoder:
    """Blocks of one encoder on one device. `blocks[i]` maps the pointer names of `B200EncoderBlock` to tensors (missing
    names are NULL) and `window` to the window side; the tensors are kept alive here and read in place."""

    def __init__(self, blocks: Sequence[dict], *, dtype: torch.dtype, dim: int, heads: int, hidden: int, ffn: int, eps: float) -> None:  # noqa: PLR0913
        self.dtype, self.dim, self.heads, self.hidden, self.ffn, self.eps = dtype, dim, heads, hidden, ffn, eps
        self._keep = [dict(b) for b in blocks]
        self.count = len(blocks)
        self.blocks = (_lib.B200EncoderBlock * max(1, self.count))()
        self.device = next((t.device for b in blocks for t in b.values() if isinstance(t, torch.Tensor)), None)
        wide = 2 * hidden if ffn == FFN_SWIGLU else hidden
        shapes = {"qkv_w": (3 * dim, dim), "qkv_b": (3 * dim,), "proj_w": (dim, dim), "fc1_w": (wide, dim), "fc1_b": (wide,), "fc2_w": (dim, hidden)}
        for entry, tensors in zip(self.blocks, blocks):
            missing = _REQUIRED - set(tensors)
            if missing:
                msg = f"encoder: a block lacks {sorted(missing)}"
                raise ValueError(msg)
            entry.window = tensors.get("window", 0)
            for name in BLOCK_TENSORS:
                t = tensors.get(name)
                if t is not None:
                    shape = shapes.get(name, (dim,))
                    if name in ("rel_pos_h", "rel_pos_w"):  # as many rows as the window's side asks for; a grid's side is known at the call
                        shape = (2 * entry.window - 1, 64) if entry.window else (*t.shape[:1], 64)
                    check_parameter(name, t, shape, torch.float32 if name.startswith("gamma") else dtype, self.device)
                    setattr(entry, name, t.data_ptr())
        self._described: dict[tuple, tuple] = {}  # geometry -> (argument description, workspace bytes)

    def describe(self, batch: int, grid: tuple[int, int], prefix: int, first: int, count: int, extra: dict) -> tuple:
        """The argument description of `count` blocks from block `first` on at a geometry, and its workspace size; `extra`: further
        scalar and pointer fields.

        Raises:
            ValueError: There are no such blocks, or the library cannot take the geometry.
        """
        if not 0 <= first <= first + count <= self.count:
            msg = f"encoder: blocks {first} .. {first + count - 1} of {self.count}"
            raise ValueError(msg)
        key = (batch, grid, prefix, first, count, tuple(sorted(extra.items())))
        found = self._described.get(key)
        if found is None:
            for b in self._keep[first : first + count]:
                for name in ("rel_pos_h", "rel_pos_w"):
                    t = b.get(name)
                    if t is not None and not b.get("window", 0) and (grid[0] != grid[1] or t.shape[0] != 2 * grid[0] - 1):
                        msg = f"encoder: {name} of {t.shape[0]} rows does not fit a grid of {grid[0]} x {grid[1]}"
                        raise ValueError(msg)
            a = _lib.B200EncoderArgs()
            a.struct_size = ctypes.sizeof(_lib.B200EncoderArgs)
            a.dtype, a.batch, a.prefix, a.eps = _DTYPES[self.dtype], batch, prefix, self.eps
            a.grid_h, a.grid_w = grid
            a.dim, a.heads, a.hidden, a.ffn = self.dim, self.heads, self.hidden, self.ffn
            a.n_blocks = count
            a.blocks = ctypes.addressof(self.blocks) + first * ctypes.sizeof(_lib.B200EncoderBlock)
            for name, value in extra.items():
                setattr(a, name, value)
            size = ctypes.c_int64(0)
            _lib.raise_for_code(_lib.library().b200_encoder_workspace(ctypes.byref(a), ctypes.byref(size)), "encoder")
            if len(self._described) >= 64:  # noqa: PLR2004
                self._described.clear()
            found = self._described[key] = (a, size.value)
        return found

    def try_describe(self, *geometry: object) -> tuple | None:
        """`describe`, or None where the library cannot take the geometry (patches of an odd side, more tokens than a launch holds):
        the model's layers then run one by one."""
        try:
            return self.describe(*geometry)
        except ValueError as e:
            _LOG.info("layer by layer: %s", e)
            return None

    def launch(self, described: tuple, device: torch.device, *, x: torch.Tensor | None = None, images: torch.Tensor | None = None,
               taps: Sequence[tuple[int, torch.Tensor]] = (), neck_out: torch.Tensor | None = None) -> None:  # fmt: skip
        """Launch a described forward on the current stream of `device`, which is the parameters'.

        Raises:
            ValueError: A tensor or the parameters are on another device.
        """
        tensors = [t for t in (x, images, neck_out, *(out for _, out in taps)) if t is not None]
        if any(t.device != device for t in tensors) or self.device not in (None, device):
            msg = f"encoder: parameters on {self.device}, tensors on {[str(t.device) for t in tensors]}, launch on {device}"
            raise ValueError(msg)
        template, size = described
        a = _lib.B200EncoderArgs.from_buffer_copy(template)
        index = device.index  # a tensor's device has one
        if index != torch.cuda.current_device():
            with torch.cuda.device(index):
                self.launch(described, device, x=x, images=images, taps=taps, neck_out=neck_out)
            return
        workspace = torch.empty(max(size, 1), dtype=torch.uint8, device=device)
        a.workspace, a.workspace_bytes = workspace.data_ptr(), size
        a.x = None if x is None else x.data_ptr()
        a.images = None if images is None else images.data_ptr()
        a.neck_out = None if neck_out is None else neck_out.data_ptr()
        if taps:
            table = (_lib.B200EncoderTap * len(taps))()
            for entry, (after, out) in zip(table, taps):
                entry.after, entry.out = after, out.data_ptr()
            a.taps, a.n_taps = ctypes.addressof(table), len(taps)
        if a.prefix + a.grid_h * a.grid_w >= _SPLIT_MIN_KEYS:
            scratch = reserve_workspace(index)
            if scratch is not None:
                a.attn_workspace, a.attn_workspace_bytes = scratch.data_ptr(), scratch.numel()
        code = _lib.library().b200_encoder_forward(ctypes.byref(a), torch._C._cuda_getCurrentRawStream(index))  # noqa: SLF001
        _lib.raise_for_code(code, "encoder")


def native_or_none(blocks: Sequence[dict], others: dict[str, tuple[torch.Tensor, tuple[int, ...]]], **geometry: object) -> NativeEncoder | None:
    """The native encoder of a model's blocks, or None where the kernels cannot take a parameter, one of the table or one of `others`
    (those a call names in its description, with their shapes): the model then runs layer by layer, and its layers take the
    parameter or say what is wrong with it."""
    try:
        native = NativeEncoder(blocks, **geometry)
        for name, (t, shape) in others.items():
            check_parameter(name, t, shape, native.dtype, native.device)
    except ValueError as e:
        _LOG.info("layer by layer: %s", e)
        return None
    return native
