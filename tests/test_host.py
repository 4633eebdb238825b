"""Host-side contract of the operator, on CPU: the checks that run before any launch, the `Flash64` and SDPA
signatures, mode resolution. Mirrors the reference's launcher tests that need no GPU
(tests/test_flash64_guard.py:29-172 monkeypatches `Flash64._run`; tests/test_kernels.py:346-392 rejects arguments)."""

from __future__ import annotations

import importlib
import re
import warnings

import pytest
import torch

import fastforks_b200 as ff
from fastforks_b200.flash64 import Flash64, check_flash64

attn_mod = importlib.import_module("fastforks_b200.attention")


def test_cpu_tensors_are_rejected_not_computed() -> None:
    q = torch.zeros(1, 2, 5, 64, dtype=torch.float16)
    with pytest.raises(ValueError, match="CUDA"):
        ff.attention(q, q, q)
    with pytest.raises(ValueError, match="CUDA"):
        ff.scaled_dot_product_attention(q, q, q)
    with pytest.raises(ValueError, match="CUDA"):
        Flash64()(q, q, q, 0.125)


@pytest.mark.parametrize(
    ("shape", "dtype", "word"),
    [((1, 2, 5, 32), torch.float16, "head dim"), ((1, 2, 5, 64), torch.float32, "float16"), ((2, 5, 64), torch.float16, "4-D")],
)
def test_check_operands_messages(shape: tuple, dtype: torch.dtype, word: str) -> None:
    q = torch.zeros(shape, dtype=dtype)
    with pytest.raises(ValueError, match=word):
        attn_mod.check_operands(q, q, q)


def test_flash64_signature_and_variants() -> None:
    assert ff.FLASH_VARIANTS == ("hh", "fh", "ff")
    with pytest.raises(ValueError, match="variant"):
        Flash64("xx")
    f = Flash64("fh", probe=3)
    assert (f.variant, f.probe, f.window) == ("fh", 3, 3)
    with pytest.raises(ValueError, match="variant"):
        Flash64._run("zz", *(torch.zeros(1, 1, 1, 64),) * 3, 1.0)  # noqa: SLF001


def test_flash64_run_is_the_single_choke_point(monkeypatch: pytest.MonkeyPatch) -> None:
    """Like the reference's guard tests, a patched `_run` sees every call with (variant, q, k, v, scale)."""
    calls = []

    def fake(variant: str, q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, scale: float) -> torch.Tensor:
        calls.append((variant, q.shape, scale))
        return torch.zeros_like(q)

    monkeypatch.setattr(Flash64, "_run", staticmethod(fake))
    q = torch.zeros(2, 7, 3, 64, dtype=torch.float16)
    out = Flash64("ff")(q, q, q, 0.5)
    assert calls == [("ff", q.shape, 0.5)]
    assert out.shape == q.shape


def test_check_flash64_needs_same_shapes(monkeypatch: pytest.MonkeyPatch) -> None:
    monkeypatch.setattr(attn_mod, "check_operands", lambda *a, **k: None)
    import fastforks_b200.flash64 as f64

    monkeypatch.setattr(f64, "check_operands", lambda *a, **k: None)
    q = torch.zeros(1, 5, 2, 64, dtype=torch.float16)
    k = torch.zeros(1, 6, 2, 64, dtype=torch.float16)
    with pytest.raises(ValueError, match="self-attention only"):
        check_flash64(q, k, k)


def test_sdpa_rejects_dropout_and_causal() -> None:
    q = torch.zeros(1, 2, 5, 64, dtype=torch.float16)
    with pytest.raises(ValueError, match="dropout"):
        ff.scaled_dot_product_attention(q, q, q, dropout_p=0.1)
    with pytest.raises(ValueError, match="causal"):
        ff.scaled_dot_product_attention(q, q, q, is_causal=True)


def test_strides_and_sizes_of_both_layouts() -> None:
    packed = torch.zeros(2, 9, 3, 4, 64, dtype=torch.float16)  # [B, N, 3, H, 64]
    q = packed.unbind(2)[0]
    assert attn_mod._sizes(q, "bnhd") == (2, 9, 4)  # noqa: SLF001
    assert attn_mod._strides(q, "bnhd") == (9 * 3 * 4 * 64, 3 * 4 * 64, 64)  # noqa: SLF001
    qs = packed.permute(2, 0, 3, 1, 4)[0]  # [B, H, N, 64] view, as in _vit_kernels
    assert attn_mod._sizes(qs, "bhnd") == (2, 9, 4)  # noqa: SLF001
    assert attn_mod._strides(qs, "bhnd") == (9 * 3 * 4 * 64, 3 * 4 * 64, 64)  # noqa: SLF001


def test_bias_view_broadcasts_without_copy() -> None:
    q = torch.zeros(2, 3, 5, 64, dtype=torch.float16)
    bias = torch.zeros(1, 3, 5, 7, dtype=torch.float16)
    view, copied = attn_mod._bias_view("bias", bias, (2, 3, 5, 7), q)  # noqa: SLF001
    assert view.stride() == (0, 35, 7, 1)
    assert view.data_ptr() == bias.data_ptr() and not copied
    view, copied = attn_mod._bias_view("bias", bias.transpose(2, 3).contiguous().transpose(2, 3), (2, 3, 5, 7), q)  # noqa: SLF001
    assert copied and view.stride(-1) == 1  # a last stride other than 1 is the one case that needs a copy
    with pytest.raises(ValueError, match="broadcast"):
        attn_mod._bias_view("bias", torch.zeros(4, 3, 5, 7, dtype=torch.float16), (2, 3, 5, 7), q)  # noqa: SLF001
    with pytest.raises(ValueError, match="float16"):
        attn_mod._bias_view("bias", torch.zeros(5, 7, dtype=torch.int32), (2, 3, 5, 7), q)  # noqa: SLF001


def test_tile_layout_pads_rows_only_where_needed() -> None:
    """The layout the kernel fetches in tiles: 16-bit, 16-byte aligned base, strides of the dimensions with more than
    one entry in multiples of 8. The reference builds its windowed blocks' bias that way itself (rows padded to a
    multiple of 8 and sliced, src/fastforks/_optimize/transformer.py:463-466)."""
    swin = torch.zeros(1, 12, 49, 56, dtype=torch.float16)[..., :49]  # the reference's `_swin_bias` layout
    assert ff.tile_layout(swin).data_ptr() == swin.data_ptr()  # taken as it is
    odd = torch.arange(2 * 3 * 5 * 7, dtype=torch.float32).reshape(2, 3, 5, 7).to(torch.bfloat16)
    padded = ff.tile_layout(odd)
    assert padded.shape == odd.shape and torch.equal(padded, odd)
    assert padded.stride() == (3 * 5 * 8, 5 * 8, 8, 1) and padded.data_ptr() % 16 == 0
    assert ff.tile_layout(padded).data_ptr() == padded.data_ptr()  # idempotent
    # fewer dims are taken as broadcast over batch and heads; the stride of a dimension of one entry does not matter
    two_d = ff.tile_layout(torch.zeros(5, 7, dtype=torch.float16))
    assert two_d.shape == (1, 1, 5, 7) and two_d.stride(2) == 8
    single_row = torch.zeros(1, 1, 1, 7, dtype=torch.float16)
    assert ff.tile_layout(single_row).data_ptr() == single_row.data_ptr()
    with pytest.raises(ValueError, match="float16 / bfloat16"):
        ff.tile_layout(torch.zeros(5, 7))
    # `attention` pads a 16-bit bias itself and reports the copy; a float32 bias is passed through for the row-wise loads
    q = torch.zeros(2, 3, 5, 64, dtype=torch.float16)
    view, copied = attn_mod._bias_view("bias", odd.half(), (2, 3, 5, 7), q, tiled=True)  # noqa: SLF001
    assert copied and view.stride(2) == 8
    view, copied = attn_mod._bias_view("bias", odd.float(), (2, 3, 5, 7), q, tiled=True)  # noqa: SLF001
    assert not copied and view.stride(2) == 7


def test_rope_table_and_contract_on_the_host() -> None:
    """`rope_table` is plain torch and runs anywhere; `rope_qk_` rejects what the kernel cannot take before any launch."""
    import numpy as np

    from oracle import rope_oracle as ro

    cs = ff.rope_table(3, 4, 100.0)
    assert cs.shape == (12, 2, 32) and cs.dtype == torch.float32
    np.testing.assert_allclose(cs.numpy(), ro.rope_table(3, 4, 100.0), rtol=0, atol=2e-6)
    with pytest.raises(ValueError, match="CUDA"):
        ff.rope_qk_(torch.zeros(1, 17, 3, 2, 64, dtype=torch.float16), cs)


def test_resolve_mode_follows_the_reference_rule(caplog: pytest.LogCaptureFixture) -> None:
    assert ff.resolve_mode("portable") == "portable"
    with pytest.raises(ValueError, match="mode"):
        ff.resolve_mode("fast")
    if not torch.cuda.is_available():
        with caplog.at_level("INFO", logger="fastforks_b200"):
            assert ff.resolve_mode("auto") == "portable"  # logged, never silent
        assert "using portable" in caplog.text
        with pytest.raises(ff.BackendUnavailableError, match="no CUDA device"):
            ff.resolve_mode("kernels")


def test_missing_library_fails_loudly(monkeypatch: pytest.MonkeyPatch, tmp_path) -> None:  # noqa: ANN001
    from fastforks_b200 import _lib

    monkeypatch.setattr(_lib, "SHARED_OBJECT", tmp_path / "absent.so")
    _lib.library.cache_clear()
    try:
        with pytest.raises(ff.KernelUnavailableError, match="not built"):
            _lib.library()
    finally:
        _lib.library.cache_clear()


def fresh_host(monkeypatch: pytest.MonkeyPatch):  # noqa: ANN201
    """`_lib` as in a process that has launched nothing yet; its caches are emptied again by the caller."""
    from fastforks_b200 import _lib

    if _lib.needs_build():
        _lib.build()
    monkeypatch.setattr(_lib, "fast", None)
    monkeypatch.setattr(_lib, "_fast_tried", False)
    _lib.host.cache_clear()
    return _lib


def test_operators_work_without_the_host_extension(monkeypatch: pytest.MonkeyPatch, tmp_path) -> None:  # noqa: ANN001
    """The extension only saves host time: missing, for another torch or not loadable it leaves a warning, once, and never an
    exception, which would come behind a launch."""
    _lib = fresh_host(monkeypatch)
    try:
        with monkeypatch.context() as m:
            m.setattr(_lib, "HOST_EXTENSION", tmp_path / "absent.so")
            with pytest.warns(RuntimeWarning, match="ctypes"):
                _lib.use_fast()
            assert _lib.fast is None
            _lib.library.cache_clear()
            _lib.library()  # which does not ask for the extension
            with warnings.catch_warnings():
                warnings.simplefilter("error")
                _lib.use_fast()
        with monkeypatch.context() as m:
            m.setattr(torch, "__version__", "1.0.0+other")
            m.setattr(_lib, "_fast_tried", False)
            assert _lib.needs_build()
            with pytest.warns(RuntimeWarning, match="this torch"):
                _lib.use_fast()
        with monkeypatch.context() as m:
            broken = tmp_path / "broken.so"
            broken.write_bytes(b"b200attn-src:" + _lib.host_hash().encode())
            m.setattr(_lib, "HOST_EXTENSION", broken)
            m.setattr(_lib, "_fast_tried", False)
            with pytest.warns(RuntimeWarning, match="cannot load"):
                _lib.use_fast()
        assert _lib.fast is None
        monkeypatch.setattr(_lib, "_fast_tried", False)
        _lib.use_fast()
        assert _lib.fast is not None
    finally:
        _lib.library.cache_clear()
        _lib.host.cache_clear()


def test_a_build_without_torch_headers_still_has_the_library(monkeypatch: pytest.MonkeyPatch, tmp_path) -> None:  # noqa: ANN001
    _lib = fresh_host(monkeypatch)
    monkeypatch.setattr(_lib, "HOST_EXTENSION", tmp_path / "_b200host.so")
    for command in (["false"], [str(tmp_path / "no-such-compiler")]):
        monkeypatch.setattr(_lib, "host_build_command", lambda *a, command=command: command)
        with pytest.warns(RuntimeWarning, match="did not compile"):
            assert _lib.build() == _lib.SHARED_OBJECT
    assert not _lib.HOST_EXTENSION.exists()


def test_host_attention_contract_is_checked_before_any_copy() -> None:
    """`HostAttention.check` is host logic only: it needs no device and rejects what the copies could not take."""
    check = ff.HostAttention.check
    x = torch.zeros(2, 5, 3, 4, 64, dtype=torch.float16)
    o = torch.zeros(2, 5, 4, 64, dtype=torch.float16)
    check([], [])
    with pytest.raises(ValueError, match="outputs"):
        check([x], [])
    with pytest.raises(ValueError, match="packed"):
        check([x[:, :, 0]], [o])
    with pytest.raises(ValueError, match="expected"):
        check([x], [o[:, :4].contiguous()])
    with pytest.raises(ValueError, match="float16"):
        check([x.float()], [o.float()])
    with pytest.raises(ValueError, match="contiguous"):
        check([x.transpose(0, 1).contiguous().transpose(0, 1)], [o])
    with pytest.raises(ValueError, match="differs"):
        check([x, torch.zeros(1, 5, 3, 4, 64, dtype=torch.float16)], [o, torch.zeros(1, 5, 4, 64, dtype=torch.float16)])
    with pytest.raises(ValueError, match="empty"):
        check([x[:0]], [o[:0]])


@pytest.mark.parametrize("native", [True, False])
def test_a_snapshot_sees_tensors_that_were_replaced(native: bool, monkeypatch: pytest.MonkeyPatch) -> None:  # noqa: FBT001
    """What an encoder's table of parameter addresses rests on: values written in place leave it valid, another tensor, other
    storage, another shape, one more or one less do not."""
    from fastforks_b200 import _lib, encoder

    monkeypatch.setattr(_lib, "fast", _lib.host() if native else None)
    monkeypatch.setattr(_lib, "_fast_tried", True)
    a = {"x": torch.zeros(4, 6), "y": torch.zeros(3, dtype=torch.float16)}
    b = {"x": torch.zeros(2)}
    snap = encoder.Snapshot(a, b)
    a["x"].add_(1.0)
    assert not snap.changed(a, b)
    assert snap.changed(a) and snap.changed(b, a) and snap.changed({**a, "z": torch.zeros(1)}, b)
    assert snap.changed({"x": a["x"].clone(), "y": a["y"]}, b) and snap.changed({"x": a["x"], "y": 3.0}, b) if native else True
    a["x"].t_()
    assert snap.changed(a, b)
    a["x"].t_()
    assert not snap.changed(a, b)
    b["x"].data = b["x"].clone()
    assert snap.changed(a, b)
    assert not encoder.Snapshot(a, b).changed(a, b)


def test_kernels_hold_their_tensor_memory_before_they_let_the_next_kernel_start() -> None:
    """A kernel that starts early allocates tensor memory in its set-up and then waits for the grid in front of it. If that grid let it
    start before all of its own CTAs had theirs, the two could wait for each other for ever (an allocation has no time limit)."""
    from fastforks_b200 import _lib

    checked = 0
    for path in (*_lib.SOURCES, *_lib.HEADERS):
        for body in path.read_text().split("__global__")[1:]:
            if "tmem_alloc" not in body or "grid_launch_dependents();" not in body:
                continue
            name = body[: body.index("(", body.index("_kernel"))].split()[-1]
            assert body.index("tmem_alloc") < body.index("grid_launch_dependents();"), f"{path.name}: {name}"
            checked += 1
    assert checked == 4  # attention, pair and split GEMM, SAM's terms by lines


def test_kernels_that_give_up_wait_for_their_products_before_they_free_tensor_memory() -> None:
    """A wait that runs out ends a kernel early. Products in flight still read its shared memory and write its tensor memory, so none may
    free that without a wait behind a last commit that looks at no abort flag; and a loop that would overwrite operands ends first.
    (Read, not run: nothing makes a wait on products run out on a healthy GPU.)"""
    from fastforks_b200 import _lib

    checked = {}
    for path in (*_lib.SOURCES, *_lib.HEADERS):
        for body in path.read_text().split("__global__")[1:]:
            if "tmem_dealloc" not in body:
                continue
            name = body[: body.index("(", body.index("_kernel"))].split()[-1]
            drained = re.search(r"umma_commit(_pair)?\(&(sm\.)?(drain(\[t\])?|acc_full)\);", body)
            assert drained, name
            assert drained.start() < body.index("tmem_dealloc"), name
            checked[name] = body
    assert len(checked) == 4  # attention, pair and split GEMM, SAM's terms by lines
    lines = checked["sam_rel_lines_kernel"]
    gives_up = lines.index("if (abort != 0)")
    assert lines.rindex("__syncthreads();", 0, gives_up) > lines.index("mbar_wait(&done")  # the flag is looked at where all warps see the same
    assert "break;" in lines[gives_up : lines.index("tmem_dealloc")]


def test_a_pair_of_ctas_waits_for_every_signal_of_the_other_before_either_goes() -> None:
    """An arrival on a barrier of a CTA that has gone hits whatever took its shared memory. The pair kernel's barrier at the end is relaxed
    and orders no such arrival, so the leader waits for those that hand accumulators back: in its loop for all but the last on either
    barrier, behind the loop for these. (Read, not run.) The phases waited for are counted here for any number of items."""
    from fastforks_b200 import _lib

    source = next(p for p in _lib.HEADERS if p.name == "gemm_sm100.cuh").read_text()
    body = next(b for b in source.split("__global__")[1:] if "gemm_pair_kernel(" in b)
    issuer = body[body.index("= MMA issuer") : body.index("= epilogue warps")]
    assert "if (it >= 2) ok = __all_sync(0xffffffffu, mbar_wait(&sm.acc_empty[it & 1], ((it >> 1) - 1) & 1, abort_flag));" in issuer
    behind = "if (ok) ok = __all_sync(0xffffffffu, lane >= min(it, 2) || mbar_wait(&sm.acc_empty[lane], ((it - 1 - lane) / 2) & 1, abort_flag));"
    assert issuer.index("umma_commit_pair(&sm.acc_full") < issuer.index(behind) < issuer.index("umma_commit_pair(&sm.drain)")
    for items in range(9):
        waited = [(it & 1, (it >> 1) - 1) for it in range(2, items)] + [(lane, (items - 1 - lane) // 2) for lane in range(min(items, 2))]
        assert sorted(waited) == sorted((it & 1, it >> 1) for it in range(items))  # every phase of both barriers, once


def test_a_stage_is_signalled_in_front_of_the_accumulator_it_is_part_of() -> None:
    """The signals of the last stages reach the other CTA ahead of the accumulator's, which all its epilogue warps wait for."""
    from fastforks_b200 import _lib

    source = next(p for p in _lib.HEADERS if p.name == "gemm_sm100.cuh").read_text()
    body = next(b for b in source.split("__global__")[1:] if "gemm_pair_kernel(" in b)
    assert body.index("umma_commit_pair(&sm.empty[st]);") < body.index("umma_commit_pair(&sm.acc_full[it & 1]);")
    assert "mbar_wait(&sm.acc_full[it & 1], (it >> 1) & 1, abort_flag)" in body


def test_a_pair_that_gives_up_waits_for_the_residuals_it_has_asked_for_and_no_others() -> None:
    """A wait for a phase that nothing will complete runs to its limit, a second each. So the drain of residual loads lies where the wait for
    them ran out, the only place where one can be on its way: under the condition they were asked for under, on the phase that wait was
    for, and the count of phases moves on behind it. (Read, not run: nothing makes that wait run out on a healthy GPU.)"""
    from fastforks_b200 import _lib

    source = next(p for p in _lib.HEADERS if p.name == "gemm_sm100.cuh").read_text()
    body = next(b for b in source.split("__global__")[1:] if "gemm_pair_kernel(" in b)
    epilogue = body[body.index("= epilogue warps") :]
    waits = [m.start() for m in re.finditer(r"mbar_wait\(&sm\.res_full\[e\]\[i\], loads\[i\] & 1, (&no_abort|abort_flag)\)", epilogue)]
    assert len(waits) == 2 == epilogue.count("mbar_wait(&sm.res_full")
    assert all(epilogue[:w].rstrip().endswith(("if (asked(i))", "if (asked(i)) ok = ok && __all_sync(0xffffffffu,")) for w in waits)
    gives_up = epilogue.index("if (!ok) {", waits[0])
    assert waits[0] < gives_up < waits[1] < epilogue.index("break;", gives_up) < epilogue.index("loads[i] += asked(i) ? 1 : 0;") < epilogue.index("mbar_wait(&sm.acc_full")
    asked = "part + 2 * i < pieces && inside(row0, col0 + (part + 2 * i) * 64)"
    assert f"auto asked = [&](int i) {{ return {asked}; }};" in epilogue
    assert re.search(r"const int c = part \+ 2 \* i;\s+if \(c < pieces && inside\(row0, col0 \+ c \* 64\)\) \{", epilogue[: waits[0]])
