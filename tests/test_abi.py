"""The C ABI without a GPU: the library loads, exports every symbol `include/b200_attn.h` declares, the ctypes
mirror of `B200AttnArgs` matches the C struct, and argument checks reject bad calls before any launch
(the reference checks the same way: signatures vs sources in tests/test_kernels.py:112-124, argument rejection
before launch in tests/test_kernels.py:346-392)."""

from __future__ import annotations

import ctypes
import re
import shutil
import subprocess
from pathlib import Path

import pytest

from fastforks_b200 import _lib

ROOT = Path(__file__).resolve().parent.parent
HEADER = ROOT / "include" / "b200_attn.h"


@pytest.fixture(scope="module")
def lib() -> ctypes.CDLL:
    if _lib.needs_build():
        _lib.build()
    _lib.library.cache_clear()
    return _lib.library()


def declared_functions() -> list[str]:
    text = re.sub(r"/\*.*?\*/", "", HEADER.read_text(), flags=re.S)
    return re.findall(r"^\s*(?:const\s+)?[\w\*]+\s+\*?\s*(b200_(?:attn|sam|gemm|rope)\w*)\s*\(", text, flags=re.M)


def test_header_declares_the_expected_entry_points() -> None:
    assert sorted(declared_functions()) == sorted(_lib.EXPORTS)


def test_library_exports_every_declared_symbol(lib: ctypes.CDLL) -> None:
    for name in declared_functions():
        assert hasattr(lib, name), name
    assert b"sm_100a" in lib.b200_attn_version()


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
def test_ctypes_struct_matches_the_c_struct(tmp_path: Path) -> None:
    fields = [name for name, *_ in _lib.B200AttnArgs._fields_]  # noqa: SLF001
    src = tmp_path / "layout.c"
    lines = "\n".join(f'  printf("{f} %zu\\n", offsetof(B200AttnArgs, {f}));' for f in fields)
    src.write_text(
        f'#include <stdio.h>\n#include <stddef.h>\n#include "{HEADER}"\n'
        f'int main(void) {{\n  printf("sizeof %zu\\n", sizeof(B200AttnArgs));\n{lines}\n  return 0;\n}}\n'
    )
    exe = tmp_path / "layout"
    subprocess.run(["gcc", "-std=c99", "-Wall", "-Werror", "-o", str(exe), str(src)], check=True)
    out = dict(line.split() for line in subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines())
    assert int(out.pop("sizeof")) == ctypes.sizeof(_lib.B200AttnArgs)
    for f in fields:
        assert int(out[f]) == getattr(_lib.B200AttnArgs, f).offset, f


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
def test_ctypes_structs_of_the_encoder_match_the_c_structs(tmp_path: Path) -> None:
    structs = (_lib.B200EncoderBlock, _lib.B200EncoderTap, _lib.B200EncoderArgs)
    want = {f"{s.__name__}.{f}": getattr(s, f).offset for s in structs for f, *_ in s._fields_}  # noqa: SLF001
    want |= {s.__name__: ctypes.sizeof(s) for s in structs}
    src = tmp_path / "layout.c"
    lines = "\n".join(f'  printf("{name} %zu\\n", {"offsetof(" + name.replace(".", ", ") + ")" if "." in name else "sizeof(" + name + ")"});' for name in want)
    src.write_text(f'#include <stdio.h>\n#include <stddef.h>\n#include "{ROOT / "include" / "b200_encoder.h"}"\nint main(void) {{\n{lines}\n  return 0;\n}}\n')
    exe = tmp_path / "layout"
    subprocess.run(["gcc", "-std=c99", "-Wall", "-Werror", "-o", str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()
    assert {name: int(offset) for name, offset in (line.split() for line in out)} == want


def _args(**kw: object) -> _lib.B200AttnArgs:
    a = _lib.B200AttnArgs()
    a.struct_size = ctypes.sizeof(_lib.B200AttnArgs)
    a.dtype = _lib.F16
    a.q = a.k = a.v = a.o = 0x10000  # only inspected for alignment by b200_attn_query
    for s in (a.q_stride, a.k_stride, a.v_stride, a.o_stride):
        s[:] = (197 * 12 * 64, 12 * 64, 64)
    a.batch, a.heads, a.q_tokens, a.kv_tokens, a.head_dim = 1, 12, 197, 197, 64
    a.scale = 0.125
    for k, v in kw.items():
        if isinstance(v, tuple):
            getattr(a, k)[:] = v
        else:
            setattr(a, k, v)
    return a


def test_query_accepts_the_reference_shapes(lib: ctypes.CDLL) -> None:
    sched = ctypes.c_int32(-1)
    assert lib.b200_attn_query(ctypes.byref(_args()), ctypes.byref(sched)) == _lib.OK
    assert sched.value in (_lib.SCHED_LONG, _lib.SCHED_SHORT)
    packed = (197 * 3 * 12 * 64, 3 * 12 * 64, 64)  # views of packed qkv [B, N, 3, H, 64]
    assert lib.b200_attn_query(ctypes.byref(_args(q_stride=packed, k_stride=packed, v_stride=packed)), None) == _lib.OK
    assert lib.b200_attn_query(ctypes.byref(_args(dtype=_lib.BF16, q_tokens=4096, kv_tokens=4096)), None) == _lib.OK


@pytest.mark.parametrize(
    ("kw", "code", "word"),
    [
        ({"struct_size": 8}, _lib.BAD_CONFIG, "struct_size"),
        ({"dtype": 7}, _lib.BAD_CONFIG, "dtype"),
        ({"head_dim": 128}, _lib.UNSUPPORTED, "head dim"),
        ({"q_tokens": 0}, _lib.UNSUPPORTED, "empty"),
        ({"kv_tokens": 0}, _lib.UNSUPPORTED, "empty"),
        ({"scale": 0.0}, _lib.UNSUPPORTED, "scale"),
        ({"scale": float("nan")}, _lib.UNSUPPORTED, "scale"),
        ({"q": 0}, _lib.BAD_CONFIG, "NULL"),
        ({"k": 0x10008}, _lib.UNSUPPORTED, "aligned"),
        ({"v_stride": (197 * 12 * 64, 12 * 64 + 4, 64)}, _lib.UNSUPPORTED, "multiple of 8"),
        ({"bias": 0x10000, "rel_h": 0x10000, "rel_w": 0x10000}, _lib.BAD_CONFIG, "exclusive"),
        ({"rel_h": 0x10000}, _lib.BAD_CONFIG, "together"),
        ({"rel_h": 0x10000, "rel_w": 0x10000, "rel_kh": 14, "rel_kw": 13}, _lib.UNSUPPORTED, "kv_tokens"),
        ({"bias": 0x10000, "bias_dtype": 9}, _lib.BAD_CONFIG, "bias_dtype"),
        ({"schedule": 5}, _lib.BAD_CONFIG, "schedule"),
    ],
)
def test_query_rejects_before_launch(lib: ctypes.CDLL, kw: dict, code: int, word: str) -> None:
    assert lib.b200_attn_query(ctypes.byref(_args(**kw)), None) == code
    assert word in lib.b200_attn_last_error().decode()


def test_fwd_rejects_bad_arguments_without_a_gpu(lib: ctypes.CDLL) -> None:
    """`b200_attn_fwd` runs the same checks first, so a bad call returns before touching the CUDA runtime."""
    assert lib.b200_attn_fwd(ctypes.byref(_args(head_dim=32)), None) == _lib.UNSUPPORTED
    assert lib.b200_attn_fwd(None, None) == _lib.BAD_CONFIG


def test_return_codes_map_to_the_reference_exceptions(lib: ctypes.CDLL) -> None:
    lib.b200_attn_query(ctypes.byref(_args(head_dim=32)), None)
    with pytest.raises(ValueError, match="head dim"):
        _lib.raise_for_code(_lib.UNSUPPORTED, "attention")
    with pytest.raises(RuntimeError):
        _lib.raise_for_code(_lib.CUDA_ERROR_BASE + 2, "attention")
    _lib.raise_for_code(_lib.OK, "attention")


def _encoder_args(**kw: object) -> _lib.B200EncoderArgs:
    """An encoder of one SAM block with images, a tap and a neck; addresses are only looked at."""
    block = (_lib.B200EncoderBlock * 1)()
    for name, kind in _lib.B200EncoderBlock._fields_:  # noqa: SLF001
        if kind is ctypes.c_void_p:
            setattr(block[0], name, kw.pop(f"block.{name}", 0x10000))
    block[0].window = kw.pop("block.window", 4)
    tap = (_lib.B200EncoderTap * 1)((0, 0, kw.pop("tap.out", 0x10000)))
    a = _lib.B200EncoderArgs()
    a.struct_size = ctypes.sizeof(_lib.B200EncoderArgs)
    a.batch, a.grid_h, a.grid_w, a.dim, a.heads, a.hidden, a.ffn, a.n_blocks = 1, 6, 6, 128, 2, 512, 2, 1
    a.blocks, a.taps, a.n_taps = ctypes.addressof(block), ctypes.addressof(tap), 1
    a.images, a.image_dtype, a.height, a.width, a.patch, a.patch_k = 0x10000, _lib.F32, 96, 96, 16, 768
    a.neck_channels, a.workspace, a.workspace_bytes = 24, 0x10000, 0
    for name in ("patch_w", "start", "patch_b", "norm_w", "norm_b", *(f"neck_{n}" for n in ("w0", "n0_w", "n0_b", "w1", "n1_w", "n1_b", "out"))):
        setattr(a, name, 0x10000)
    for name, value in kw.items():
        setattr(a, name, value)
    a.keep = block, tap
    return a


ENCODER_POINTERS = {"patch_w": True, "start": True, "patch_b": False, "first": False, "norm_w": True, "norm_b": True, "images": None, "x": False, "tap.out": True,
                    "neck_n0_w": True, "neck_n0_b": True, "neck_w1": True, "neck_n1_w": True, "neck_n1_b": True, "neck_out": True,
                    **{f"block.{n}": n.startswith(("norm", "rel")) or n.endswith("_w") for n, k in _lib.B200EncoderBlock._fields_ if k is ctypes.c_void_p}}  # fmt: skip


@pytest.mark.parametrize("name", ENCODER_POINTERS)
def test_encoder_forward_looks_at_every_address(lib: ctypes.CDLL, name: str) -> None:
    """A NULL where something is read and an address off a 16-byte boundary are refused before the first launch."""
    forward = lambda **kw: lib.b200_encoder_forward(ctypes.byref(_encoder_args(**kw)), None)  # noqa: E731
    assert forward() == _lib.BAD_CONFIG and "workspace" in lib.b200_attn_last_error().decode()  # everything else is accepted
    assert forward(**{name: 0x10008}) == _lib.UNSUPPORTED
    assert name.removeprefix("block.").removeprefix("tap.") in lib.b200_attn_last_error().decode()
    if ENCODER_POINTERS[name]:
        assert forward(**{name: None}) in (_lib.BAD_CONFIG, _lib.UNSUPPORTED) and "workspace" not in lib.b200_attn_last_error().decode()
    elif ENCODER_POINTERS[name] is False:
        assert forward(**{name: None}) == _lib.BAD_CONFIG and "workspace" in lib.b200_attn_last_error().decode()


@pytest.mark.parametrize("window", [128, 5, 40000, 1 << 20, (1 << 31) - 1])
def test_encoder_refuses_windows_it_cannot_count(lib: ctypes.CDLL, window: int) -> None:
    """Padded windows hold more rows than the grid: their number must fit the kernels' 32-bit row numbers too. Sides the
    relative terms do not take are refused before the first launch, not between two of them."""
    size = ctypes.c_int64(0)
    plain = {"block.rel_pos_h": None, "block.rel_pos_w": None}
    assert lib.b200_encoder_workspace(ctypes.byref(_encoder_args(**{"block.window": 4})), ctypes.byref(size)) == _lib.OK
    assert lib.b200_encoder_workspace(ctypes.byref(_encoder_args(**{"block.window": window})), ctypes.byref(size)) == _lib.UNSUPPORTED
    want = _lib.OK if window < 1000 else _lib.UNSUPPORTED  # noqa: PLR2004
    assert lib.b200_encoder_workspace(ctypes.byref(_encoder_args(**{"block.window": window}, **plain)), ctypes.byref(size)) == want


def test_gemm_plan_on_the_host(lib: ctypes.CDLL) -> None:
    """The plan as a function of sizes and of the device's description, without a GPU."""
    clusters, plan = (ctypes.c_int32 * 6)(148, 74, 48, 36, 22, 16), (ctypes.c_int32 * 3)()
    seen = {}
    for shape in ((197, 768, 3072), (100, 72, 8), (5480, 4096, 1024), (21920, 1536, 4096), (2740, 4096, 200)):
        assert lib.b200_gemm_plan(*shape, 148, clusters, plan) == _lib.OK
        seen[shape] = tuple(plan)
    assert seen[197, 768, 3072][1] > 1  # few tiles: the k range is shared
    assert seen[100, 72, 8] == (64, 1, 0)
    assert seen[5480, 4096, 1024][:2] == seen[21920, 1536, 4096][:2] == (256, 0)
    assert seen[2740, 4096, 200] == (256, 0, 128)  # 176 tiles on 74 pairs: the last round in halves
    none = (ctypes.c_int32 * 6)(148, 0, 0, 0, 0, 0)  # a device that runs no clusters of the split kernel
    assert lib.b200_gemm_plan(197, 768, 3072, 148, none, plan) == _lib.OK and plan[1] <= 1
    assert lib.b200_gemm_plan(0, 8, 8, 148, clusters, plan) == lib.b200_gemm_plan(8, 8, 8, 148, None, plan) == _lib.BAD_CONFIG
