"""Loader and in-tree build of `libb200attn.so`, the C-ABI attention library declared in `include/b200_attn.h`.

The library is loaded with ctypes, the way the reference loads its `shared`-kind kernel libraries
(`src/fastforks/_core/kernels.py:481-494`): plain pointers and sizes go in, a status code comes back, and the
launch goes to torch's current raw stream (`src/fastforks/_core/kernels.py:426-428`).
"""

from __future__ import annotations

import ctypes
import functools
import hashlib
import importlib.machinery
import importlib.util
import os
import re
import shutil
import subprocess
import sys
import tempfile
import threading
import warnings
from pathlib import Path
from typing import TYPE_CHECKING

from .errors import KernelUnavailableError

if TYPE_CHECKING:
    from types import ModuleType

LIBRARY = "b200attn"
PACKAGE_DIR = Path(__file__).resolve().parent
SOURCES = tuple(PACKAGE_DIR / "csrc" / name for name in ("b200_attn.cu", "b200_window.cu", "b200_linear.cu", "b200_encoder.cu"))
HEADERS = (
    PACKAGE_DIR / "csrc" / "host_common.h",
    PACKAGE_DIR / "csrc" / "linear_host.h",
    PACKAGE_DIR / "csrc" / "sm100_ptx.cuh",
    PACKAGE_DIR / "csrc" / "attn_fwd_sm100.cuh",
    PACKAGE_DIR / "csrc" / "attn_small_sm100.cuh",
    PACKAGE_DIR / "csrc" / "attn_window_sm100.cuh",
    PACKAGE_DIR / "csrc" / "window_host.h",
    PACKAGE_DIR / "csrc" / "sam_rel_terms.cuh",
    PACKAGE_DIR / "csrc" / "rope_sm100.cuh",
    PACKAGE_DIR / "csrc" / "gemm_sm100.cuh",
    PACKAGE_DIR / "csrc" / "encoder_kernels.cuh",
    PACKAGE_DIR.parent / "include" / "b200_attn.h",
    PACKAGE_DIR.parent / "include" / "b200_encoder.h",
)
SHARED_OBJECT = PACKAGE_DIR / "libb200attn.so"
# The host side of repeated calls, a CPython extension over torch's C++ interface (no kernels in it).
HOST_SOURCE = PACKAGE_DIR / "csrc" / "host_ext.cpp"
HOST_EXTENSION = PACKAGE_DIR / "_b200host.so"

# sm_100a only: the kernels use tcgen05 / TMEM / TMA, which exist in no other target.
NVCC_FLAGS = (
    "-gencode", "arch=compute_100a,code=sm_100a", "-lineinfo", "-O3", "-std=c++17", "--expt-relaxed-constexpr",
    "-Xcompiler", "-fPIC",
)  # fmt: skip

# Every symbol include/b200_attn.h declares.
EXPORTS = (
    "b200_attn_fwd", "b200_attn_fwd_static", "b200_gemm", "b200_gemm_plan", "b200_sam_rel_terms", "b200_rope_qk", "b200_attn_query", "b200_attn_plan", "b200_attn_workspace_size", "b200_attn_status",
    "b200_attn_selftest_wait_limit", "b200_attn_last_error", "b200_attn_version",
)  # fmt: skip

# ... and include/b200_encoder.h.
ENCODER_EXPORTS = ("b200_encoder_workspace", "b200_encoder_forward")

OK, UNSUPPORTED, BAD_CONFIG, CUDA_ERROR_BASE = 0, 1, -1, 1000
F16, BF16, F32 = 0, 1, 2
SCHED_AUTO, SCHED_LONG, SCHED_SHORT = 0, 1, 2


class B200AttnArgs(ctypes.Structure):
    """Mirror of `struct B200AttnArgs` (include/b200_attn.h)."""

    _fields_ = (
        ("struct_size", ctypes.c_uint32),
        ("dtype", ctypes.c_uint32),
        ("q", ctypes.c_void_p),
        ("k", ctypes.c_void_p),
        ("v", ctypes.c_void_p),
        ("o", ctypes.c_void_p),
        ("q_stride", ctypes.c_int64 * 3),
        ("k_stride", ctypes.c_int64 * 3),
        ("v_stride", ctypes.c_int64 * 3),
        ("o_stride", ctypes.c_int64 * 3),
        ("batch", ctypes.c_int32),
        ("heads", ctypes.c_int32),
        ("q_tokens", ctypes.c_int32),
        ("kv_tokens", ctypes.c_int32),
        ("head_dim", ctypes.c_int32),
        ("scale", ctypes.c_float),
        ("bias", ctypes.c_void_p),
        ("bias_dtype", ctypes.c_uint32),
        ("bias_stride", ctypes.c_int64 * 3),
        ("rel_h", ctypes.c_void_p),
        ("rel_w", ctypes.c_void_p),
        ("rel_dtype", ctypes.c_uint32),
        ("rel_kh", ctypes.c_int32),
        ("rel_kw", ctypes.c_int32),
        ("rel_h_stride", ctypes.c_int64 * 3),
        ("rel_w_stride", ctypes.c_int64 * 3),
        ("schedule", ctypes.c_int32),
        ("test_flags", ctypes.c_int32),
        ("workspace", ctypes.c_void_p),
        ("workspace_bytes", ctypes.c_int64),
    )


class B200GemmArgs(ctypes.Structure):
    """Mirror of `struct B200GemmArgs` (include/b200_attn.h)."""

    _fields_ = (
        ("struct_size", ctypes.c_uint32),
        ("dtype", ctypes.c_uint32),
        ("m", ctypes.c_int32),
        ("n", ctypes.c_int32),
        ("k", ctypes.c_int32),
        ("act", ctypes.c_int32),
        ("x", ctypes.c_void_p),
        ("lda", ctypes.c_int64),
        ("w", ctypes.c_void_p),
        ("bias", ctypes.c_void_p),
        ("scale", ctypes.c_void_p),
        ("res", ctypes.c_void_p),
        ("lres", ctypes.c_int64),
        ("y", ctypes.c_void_p),
        ("ldy", ctypes.c_int64),
    )


class B200RelTermsArgs(ctypes.Structure):
    """Mirror of `struct B200RelTermsArgs` (include/b200_attn.h)."""

    _fields_ = (
        ("struct_size", ctypes.c_uint32),
        ("dtype", ctypes.c_uint32),
        ("q", ctypes.c_void_p),
        ("q_stride", ctypes.c_int64 * 3),
        ("rel_pos_h", ctypes.c_void_p),
        ("rel_pos_w", ctypes.c_void_p),
        ("rel_h", ctypes.c_void_p),
        ("rel_w", ctypes.c_void_p),
        ("batch", ctypes.c_int32),
        ("heads", ctypes.c_int32),
        ("side", ctypes.c_int32),
        ("head_dim", ctypes.c_int32),
    )


class B200RopeArgs(ctypes.Structure):
    """Mirror of `struct B200RopeArgs` (include/b200_attn.h)."""

    _fields_ = (
        ("struct_size", ctypes.c_uint32),
        ("dtype", ctypes.c_uint32),
        ("q", ctypes.c_void_p),
        ("k", ctypes.c_void_p),
        ("q_stride", ctypes.c_int64 * 3),
        ("k_stride", ctypes.c_int64 * 3),
        ("cs", ctypes.c_void_p),
        ("batch", ctypes.c_int32),
        ("heads", ctypes.c_int32),
        ("tokens", ctypes.c_int32),
        ("prefix", ctypes.c_int32),
        ("head_dim", ctypes.c_int32),
        ("q_scale", ctypes.c_float),
    )


class B200EncoderBlock(ctypes.Structure):
    """Mirror of `struct B200EncoderBlock` (include/b200_encoder.h)."""

    _fields_ = (
        ("norm1_w", ctypes.c_void_p),
        ("norm1_b", ctypes.c_void_p),
        ("qkv_w", ctypes.c_void_p),
        ("qkv_b", ctypes.c_void_p),
        ("proj_w", ctypes.c_void_p),
        ("proj_b", ctypes.c_void_p),
        ("gamma1", ctypes.c_void_p),
        ("norm2_w", ctypes.c_void_p),
        ("norm2_b", ctypes.c_void_p),
        ("fc1_w", ctypes.c_void_p),
        ("fc1_b", ctypes.c_void_p),
        ("fc2_w", ctypes.c_void_p),
        ("fc2_b", ctypes.c_void_p),
        ("gamma2", ctypes.c_void_p),
        ("rel_pos_h", ctypes.c_void_p),
        ("rel_pos_w", ctypes.c_void_p),
        ("window", ctypes.c_int32),
        ("reserved", ctypes.c_int32),
    )


class B200EncoderTap(ctypes.Structure):
    """Mirror of `struct B200EncoderTap` (include/b200_encoder.h)."""

    _fields_ = (("after", ctypes.c_int32), ("reserved", ctypes.c_int32), ("out", ctypes.c_void_p))


class B200EncoderArgs(ctypes.Structure):
    """Mirror of `struct B200EncoderArgs` (include/b200_encoder.h)."""

    _fields_ = (
        ("struct_size", ctypes.c_uint32),
        ("dtype", ctypes.c_uint32),
        ("batch", ctypes.c_int32),
        ("grid_h", ctypes.c_int32),
        ("grid_w", ctypes.c_int32),
        ("prefix", ctypes.c_int32),
        ("dim", ctypes.c_int32),
        ("heads", ctypes.c_int32),
        ("hidden", ctypes.c_int32),
        ("ffn", ctypes.c_int32),
        ("eps", ctypes.c_float),
        ("n_blocks", ctypes.c_int32),
        ("blocks", ctypes.c_void_p),
        ("images", ctypes.c_void_p),
        ("image_dtype", ctypes.c_uint32),
        ("height", ctypes.c_int32),
        ("width", ctypes.c_int32),
        ("patch", ctypes.c_int32),
        ("patch_w", ctypes.c_void_p),
        ("patch_k", ctypes.c_int32),
        ("n_taps", ctypes.c_int32),
        ("start", ctypes.c_void_p),
        ("x", ctypes.c_void_p),
        ("norm_w", ctypes.c_void_p),
        ("norm_b", ctypes.c_void_p),
        ("taps", ctypes.c_void_p),
        ("workspace", ctypes.c_void_p),
        ("workspace_bytes", ctypes.c_int64),
        ("attn_workspace", ctypes.c_void_p),
        ("attn_workspace_bytes", ctypes.c_int64),
        ("neck_w0", ctypes.c_void_p),
        ("neck_n0_w", ctypes.c_void_p),
        ("neck_n0_b", ctypes.c_void_p),
        ("neck_w1", ctypes.c_void_p),
        ("neck_n1_w", ctypes.c_void_p),
        ("neck_n1_b", ctypes.c_void_p),
        ("neck_out", ctypes.c_void_p),
        ("neck_channels", ctypes.c_int32),
        ("neck_eps", ctypes.c_float),
        ("patch_b", ctypes.c_void_p),
        ("first", ctypes.c_void_p),
        ("start_f32", ctypes.c_int32),
        ("patch_w_raw", ctypes.c_int32),
        ("neck_w1_conv", ctypes.c_int32),
        ("reserved", ctypes.c_int32),
    )


def source_hash() -> str:
    """Digest of the sources the shared object is compiled from (16 hex digits). The build passes it to the compiler,
    which puts it into the library's version string, so a binary can be matched with the sources beside it."""
    digest = hashlib.sha256()
    for path in sorted((*SOURCES, *HEADERS, HOST_SOURCE), key=lambda f: f.name):
        digest.update(path.name.encode())
        digest.update(path.read_bytes())
    return digest.hexdigest()[:16]


_HASH_IN_BINARY = re.compile(rb"b200attn-src:([0-9a-f]{16})")


def built_hash(binary: Path | None = None) -> str | None:
    """The source digest compiled into a binary on disk (default: the library; read from the file, without loading it), or None."""
    binary = SHARED_OBJECT if binary is None else binary
    if not binary.exists():
        return None
    found = _HASH_IN_BINARY.search(binary.read_bytes())
    return found.group(1).decode() if found else None


def host_hash() -> str:
    """Digest of what the host extension depends on: the sources, and the torch and the interpreter whose C++ and C interfaces are
    compiled into it (layouts that a binary for another version would silently get wrong)."""
    import torch  # noqa: PLC0415

    parts = (source_hash(), torch.__version__, str(torch._C._GLIBCXX_USE_CXX11_ABI), str(sys.implementation.cache_tag))  # noqa: SLF001
    return hashlib.sha256("|".join(parts).encode()).hexdigest()[:16]


def needs_build() -> bool:
    """True when a binary is missing or was compiled from other sources, or (the host extension) for another torch or Python, than
    the ones beside it."""
    return built_hash() != source_hash() or built_hash(HOST_EXTENSION) != host_hash()


def host_build_command(output: Path, digest: str) -> list[str]:
    """The compiler call for the host extension; it links against the library beside it."""
    import sysconfig  # noqa: PLC0415

    import torch  # noqa: PLC0415

    root = Path(torch.__file__).parent
    cuda = Path(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc").resolve().parent.parent
    return [
        shutil.which("g++") or "g++", "-O2", "-std=c++17", "-fPIC", "-shared", f'-DB200_SOURCE_HASH="{digest}"',
        f"-D_GLIBCXX_USE_CXX11_ABI={int(torch._C._GLIBCXX_USE_CXX11_ABI)}",  # noqa: SLF001
        f"-I{root / 'include'}", f"-I{root / 'include/torch/csrc/api/include'}", f"-I{cuda / 'include'}", f"-I{sysconfig.get_paths()['include']}",
        str(HOST_SOURCE), "-o", str(output), f"-L{PACKAGE_DIR}", "-l:libb200attn.so", "-Wl,-rpath,$ORIGIN",
        f"-L{root / 'lib'}", "-ltorch_python", "-ltorch_cuda", "-ltorch_cpu", "-ltorch", "-lc10_cuda", "-lc10", f"-Wl,-rpath,{root / 'lib'}",
    ]  # fmt: skip


_LOCK = threading.Lock()


def build(*, force: bool = False, verbose: bool = False) -> Path:
    """Compile the sources in `csrc/` for sm_100a (one compiler process each, in parallel) and link them into
    `libb200attn.so` next to this file (needs nvcc, no GPU), then the host extension. The extension only saves host time: if it does
    not compile (no torch headers), a warning says so and the library is complete without it.

    Raises:
        KernelUnavailableError: nvcc is missing or the compilation of the library failed.
    """
    with _LOCK:
        if force or built_hash() != source_hash():
            _build_library(verbose=verbose)
        if force or built_hash(HOST_EXTENSION) != host_hash():
            _build_host()
    return SHARED_OBJECT


def _build_library(*, verbose: bool) -> None:
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        raise KernelUnavailableError(LIBRARY, "nvcc not found: cannot build libb200attn.so")
    flags = [*NVCC_FLAGS, f'-DB200_SOURCE_HASH="{source_hash()}"', *(("-Xptxas", "-v") if verbose else ())]
    with tempfile.TemporaryDirectory(prefix="b200attn-") as scratch:
        objects = [Path(scratch) / f"{source.stem}.o" for source in SOURCES]
        jobs = [subprocess.Popen([nvcc, *flags, "-c", "-o", str(o), str(source)], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
                for source, o in zip(SOURCES, objects, strict=True)]  # fmt: skip
        for text, code in [(job.communicate()[0], job.returncode) for job in jobs]:
            if code != 0:
                raise KernelUnavailableError(LIBRARY, f"nvcc failed:\n{text}")
            if verbose:
                print(text)
        tmp = SHARED_OBJECT.with_suffix(f".{os.getpid()}.tmp.so")
        proc = subprocess.run([nvcc, "-shared", *NVCC_FLAGS[:2], "-o", str(tmp), *map(str, objects)], capture_output=True, text=True, check=False)
        if proc.returncode != 0:
            tmp.unlink(missing_ok=True)
            raise KernelUnavailableError(LIBRARY, f"linking failed:\n{proc.stdout}\n{proc.stderr}")
    tmp.replace(SHARED_OBJECT)


def _build_host() -> None:
    tmp = HOST_EXTENSION.with_suffix(f".{os.getpid()}.tmp.so")
    try:
        proc = subprocess.run(host_build_command(tmp, host_hash()), capture_output=True, text=True, check=False)
        text = None if proc.returncode == 0 else f"{proc.stdout}\n{proc.stderr}"
    except OSError as e:  # no compiler
        text = str(e)
    if text is None:
        tmp.replace(HOST_EXTENSION)
        return
    tmp.unlink(missing_ok=True)
    warnings.warn(f"{HOST_EXTENSION.name} did not compile: calls go through ctypes, some microseconds slower each.\n{text}", RuntimeWarning, stacklevel=3)


@functools.cache
def library() -> ctypes.CDLL:
    """The loaded `libb200attn.so` with argument types set.

    Raises:
        KernelUnavailableError: The shared object is not built or does not load (the message says which).
    """
    if built_hash() != source_hash():
        # A binary of other sources must never answer for these, and nothing is built behind the caller's back.
        state = "is not built" if not SHARED_OBJECT.exists() else "was built from other sources than the ones beside it"
        how = "run `python -c 'import fastforks_b200; fastforks_b200.build()'`"
        raise KernelUnavailableError(LIBRARY, f"{SHARED_OBJECT.name} {state}; {how}")
    try:
        lib = ctypes.CDLL(str(SHARED_OBJECT))
    except OSError as e:
        raise KernelUnavailableError(LIBRARY, f"cannot load {SHARED_OBJECT.name}: {e}") from e
    missing = [name for name in (*EXPORTS, *ENCODER_EXPORTS) if not hasattr(lib, name)]
    if missing:
        raise KernelUnavailableError(LIBRARY, f"{SHARED_OBJECT.name} lacks the symbols {missing}")
    lib.b200_attn_fwd.argtypes = (ctypes.POINTER(B200AttnArgs), ctypes.c_void_p)
    lib.b200_attn_fwd.restype = ctypes.c_int
    lib.b200_attn_fwd_static.argtypes = (ctypes.POINTER(B200AttnArgs), ctypes.c_void_p)
    lib.b200_attn_fwd_static.restype = ctypes.c_int
    lib.b200_gemm.argtypes = (ctypes.POINTER(B200GemmArgs), ctypes.c_void_p)
    lib.b200_gemm.restype = ctypes.c_int
    lib.b200_sam_rel_terms.argtypes = (ctypes.POINTER(B200RelTermsArgs), ctypes.c_void_p)
    lib.b200_sam_rel_terms.restype = ctypes.c_int
    lib.b200_rope_qk.argtypes = (ctypes.POINTER(B200RopeArgs), ctypes.c_void_p)
    lib.b200_rope_qk.restype = ctypes.c_int
    lib.b200_encoder_workspace.argtypes = (ctypes.POINTER(B200EncoderArgs), ctypes.POINTER(ctypes.c_int64))
    lib.b200_encoder_workspace.restype = ctypes.c_int
    lib.b200_encoder_forward.argtypes = (ctypes.POINTER(B200EncoderArgs), ctypes.c_void_p)
    lib.b200_encoder_forward.restype = ctypes.c_int
    lib.b200_attn_query.argtypes = (ctypes.POINTER(B200AttnArgs), ctypes.POINTER(ctypes.c_int32))
    lib.b200_attn_query.restype = ctypes.c_int
    i32p = ctypes.POINTER(ctypes.c_int32)
    lib.b200_attn_plan.argtypes = (ctypes.POINTER(B200AttnArgs), ctypes.c_int32, ctypes.c_int32, i32p, i32p, ctypes.c_int32, i32p, i32p)
    lib.b200_attn_plan.restype = ctypes.c_int
    lib.b200_gemm_plan.argtypes = (ctypes.c_int32, ctypes.c_int32, ctypes.c_int32, ctypes.c_int32, i32p, i32p)
    lib.b200_gemm_plan.restype = ctypes.c_int
    lib.b200_attn_workspace_size.argtypes = (ctypes.POINTER(ctypes.c_int64),)
    lib.b200_attn_workspace_size.restype = ctypes.c_int
    lib.b200_attn_status.argtypes = (ctypes.POINTER(ctypes.c_uint32),)
    lib.b200_attn_status.restype = ctypes.c_int
    lib.b200_attn_selftest_wait_limit.argtypes = (ctypes.c_uint32, ctypes.c_void_p)
    lib.b200_attn_selftest_wait_limit.restype = ctypes.c_int
    lib.b200_attn_last_error.argtypes = ()
    lib.b200_attn_last_error.restype = ctypes.c_char_p
    lib.b200_attn_version.argtypes = ()
    lib.b200_attn_version.restype = ctypes.c_char_p
    return lib


@functools.cache
def host() -> ModuleType:
    """The loaded host extension.

    Raises:
        KernelUnavailableError: The library or the extension is not built for these sources, this torch and this Python, or does not
            load.
    """
    library()
    if built_hash(HOST_EXTENSION) != host_hash():
        raise KernelUnavailableError(LIBRARY, f"{HOST_EXTENSION.name} is not built for these sources, this torch and this Python")
    loader = importlib.machinery.ExtensionFileLoader("_b200host", str(HOST_EXTENSION))
    spec = importlib.util.spec_from_file_location("_b200host", str(HOST_EXTENSION), loader=loader)
    try:
        module = importlib.util.module_from_spec(spec)
        loader.exec_module(module)
    except ImportError as e:
        raise KernelUnavailableError(LIBRARY, f"cannot load {HOST_EXTENSION.name}: {e}") from e
    return module


# The host extension, once this process has launched an operator the full way (the library is loaded and checked then). Its
# functions take the plain, valid call of an operator and answer None (False) to anything else.
fast: ModuleType | None = None
_fast_tried = False


def use_fast() -> None:
    """Let repeated calls go through the host extension. Without it every call goes through ctypes, so this never raises (it is
    called behind a launch): a warning says once that calls are slower than they could be."""
    global fast, _fast_tried  # noqa: PLW0603
    if not _fast_tried:
        _fast_tried = True
        try:
            fast = host()
        except KernelUnavailableError as e:
            warnings.warn(f"calls go through ctypes, some microseconds slower each: {e}", RuntimeWarning, stacklevel=3)


def last_error() -> str:
    """Reason of the calling thread's last non-zero return code."""
    return library().b200_attn_last_error().decode()


def raise_for_code(code: int, what: str) -> None:
    """Map a non-zero return code to the exception the reference raises for it.

    `ValueError` for geometry / configuration the kernels cannot take, `RuntimeError` for CUDA errors
    (`src/fastforks/kernels/dpt_fused/__init__.py:101-106`).
    """
    if code == OK:
        return
    msg = f"{what}: {last_error()} (code {code})"
    if code in (UNSUPPORTED, BAD_CONFIG):
        raise ValueError(msg)
    raise RuntimeError(msg)
