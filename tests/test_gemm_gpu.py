"""Parity of the fused-epilogue GEMM (`b200_gemm`, through `fastforks_b200.gemm`) with its CPU oracle on a B200.

The oracle (`oracle/gemm_oracle.py`) restates the epilogue formula of the reference's `dpt_fused` GEMMs and is pinned
to torch's `F.linear` / `F.gelu` / residual arithmetic by `tests/test_oracle.py`. Operands are rounded to 16 bits
first, accumulation is fp32 on both sides and the result is rounded to 16 bits once, so the bar is the reference's
relative form for this library's GEMMs: `|got - ref| <= 2e-2 * max|ref|`, mean within 2e-3 of that scale
(`conftest.assert_close`, reference tests/test_kernel_fuzz.py:63-83).
"""

from __future__ import annotations

import ctypes

import pytest
import torch

import fastforks_b200 as ff
from conftest import assert_close
from fastforks_b200 import _lib
from oracle import gemm_oracle as go

pytestmark = pytest.mark.gpu
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


@pytest.fixture(autouse=True)
def _kernels_ran_to_the_end():  # noqa: ANN202
    yield
    assert ff.device_status() == 0


def operands(m: int, n: int, k: int, dtype: torch.dtype, seed: int):  # noqa: ANN201
    gen = torch.Generator().manual_seed(seed)
    x = torch.randn(m, k, generator=gen).to(dtype)
    w = (torch.randn(n, k, generator=gen) * k**-0.5).to(dtype)
    bias = torch.randn(n, generator=gen).to(dtype)
    scale = torch.rand(n, generator=gen) + 0.5
    res = torch.randn(m, n, generator=gen).to(dtype)
    return x, w, bias, scale, res


def check(got: torch.Tensor, x, w, bias=None, scale=None, res=None, act: int = 0, what: str = "") -> None:  # noqa: ANN001, PLR0913
    f = lambda t: None if t is None else t.float().cpu().numpy()  # noqa: E731
    ref = go.gemm_epilogue(f(x), f(w), f(bias), f(scale), f(res), act)
    assert_close(got.float().cpu().numpy(), ref, unit_scale=False, what=what)


# tile edges (128 x 64 and 256 x 64 .. 256 tiles), k tails, the smallest problem, ViT shapes
SHAPES = [(1, 8, 8), (128, 128, 64), (129, 136, 72), (255, 256, 64), (257, 264, 200), (300, 1000, 520), (1370, 1152, 384),
          (5480, 1024, 1024), (2740, 3072, 1024), (700, 4096, 1024)]  # fmt: skip


@pytest.mark.parametrize(("m", "n", "k"), SHAPES)
@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
def test_linear_with_bias(m: int, n: int, k: int, dtype: str) -> None:
    x, w, bias, _, _ = (t.cuda() for t in operands(m, n, k, DTYPES[dtype], seed=m + n))
    out = torch.full((m, n), float("nan"), dtype=DTYPES[dtype], device="cuda")
    got = ff.gemm(x, w, bias, out=out)
    assert got is out and bool(torch.isfinite(out).all())
    check(got, x, w, bias, what=f"[{m},{n},{k}] {dtype}")


@pytest.mark.parametrize("act", [ff.ACT_RELU, ff.ACT_GELU, ff.ACT_GELU_TANH])
@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
def test_activations(act: int, dtype: str) -> None:
    x, w, bias, _, _ = (t.cuda() for t in operands(777, 520, 264, DTYPES[dtype], seed=act))
    check(ff.gemm(x, w, bias, act=act), x, w, bias, act=act, what=f"act {act} {dtype}")


@pytest.mark.parametrize(("m", "n", "k"), [(1, 16, 8), (9500, 2056, 72)])  # the split and the pair kernel
@pytest.mark.parametrize("act", [ff.ACT_GELU, ff.ACT_GELU_TANH])
def test_activations_at_the_ends_of_the_range(act: int, m: int, n: int, k: int) -> None:
    """Infinities, NaN and the largest finite values give what torch's GELU gives (a product of zeros, the values as bias)."""
    bias = torch.zeros(n)
    big = torch.finfo(torch.bfloat16).max
    bias[:8] = torch.tensor([float("inf"), -float("inf"), float("nan"), big, -big, 1e20, -1e20, -200.0])
    bias = bias.bfloat16().cuda()
    got = ff.gemm(torch.zeros(m, k, dtype=torch.bfloat16, device="cuda"), torch.zeros(n, k, dtype=torch.bfloat16, device="cuda"), bias, act=act)
    want = torch.nn.functional.gelu(bias.float(), approximate="tanh" if act == ff.ACT_GELU_TANH else "none").bfloat16()
    assert torch.equal(got.nan_to_num(nan=7.0, posinf=8.0, neginf=9.0), want.expand(m, n).nan_to_num(nan=7.0, posinf=8.0, neginf=9.0)), (got[0, :8], want[:8])


@pytest.mark.parametrize(("m", "n", "k"), [(300, 264, 136), (5480, 1024, 4096), (1370, 1536, 1536)])
@pytest.mark.parametrize("dtype", ["fp16", "bf16"])
def test_layerscale_and_in_place_residual(m: int, n: int, k: int, dtype: str) -> None:
    """`x += gamma * (o @ W^T + b)` as one call: scale = gamma (fp32), res = out = x, the block-output form of the
    reference's fused path (src/fastforks/shared/depth_anything_v2/fast_vit.py:199-208)."""
    x, w, bias, scale, res = (t.cuda() for t in operands(m, n, k, DTYPES[dtype], seed=k))
    before = res.clone()
    got = ff.gemm(x, w, bias, scale=scale, res=res, out=res)
    assert got.data_ptr() == res.data_ptr()
    check(got, x, w, bias, scale, before, what=f"in place [{m},{n},{k}] {dtype}")
    other = ff.gemm(x, w, None, res=before, act=ff.ACT_RELU)  # no bias, residual into a new tensor, then relu
    check(other, x, w, None, None, before, act=ff.ACT_RELU, what="no bias + residual + relu")


@pytest.mark.parametrize(("m", "n", "k"), [(129, 72, 72), (2740, 776, 264), (9500, 2056, 72)])  # the split kernel and two pair tiles, ragged
@pytest.mark.parametrize("act", [0, ff.ACT_RELU, ff.ACT_GELU, ff.ACT_GELU_TANH])
@pytest.mark.parametrize("scaled", [False, True])
def test_residual_and_scale_each_alone(scaled: bool, act: int, m: int, n: int, k: int) -> None:
    """A residual without a scale and a scale without a residual, with every activation (each a form of the pair kernel's epilogue)."""
    x, w, bias, scale, res = (t.cuda() for t in operands(m, n, k, torch.float16, seed=m + act))
    extra = {"scale": scale} if scaled else {"res": res}
    out = torch.full((m, n), float("nan"), dtype=torch.float16, device="cuda")
    check(ff.gemm(x, w, bias, act=act, out=out, **extra), x, w, bias, act=act, what=f"[{m},{n},{k}] act {act}", **extra)


@pytest.mark.parametrize(("m", "n", "k"), [(1500, 10240, 72), (1500, 10248, 72), (4400, 10504, 40)])
def test_raster_groups_of_narrow_and_wide_products(m: int, n: int, k: int) -> None:
    """Both sides of the width from which sixteen row tiles share a column of tiles; fewer and more row tiles than that."""
    x, w, bias, _, _ = (t.cuda() for t in operands(m, n, k, torch.float16, seed=n))
    out = torch.full((m, n), float("nan"), dtype=torch.float16, device="cuda")
    check(ff.gemm(x, w, bias, out=out), x, w, bias, what=f"[{m},{n},{k}]")


# One shape for every way a product is cut: the split kernel whole and with 2, 3, 4, 6 and 8 CTAs per cluster (uneven k
# shares, rows that do not divide, a last tile of one row), pair tiles of 64 to 256 columns, and a last round in parts.
PLANS = [(100, 72, 8), (197, 2304, 776), (257, 1024, 1544), (129, 776, 1000), (60, 64, 3080), (255, 384, 1536), (1, 8, 4096), (1000, 3000, 72),
         (1500, 768, 768), (1025, 2056, 136), (5480, 1000, 328), (9500, 2056, 72), (2740, 4096, 200), (29, 664, 264), (377, 32, 360), (20682, 8, 248),
         (5180, 728, 104), (4349, 2912, 512), (10380, 5496, 568)]  # fmt: skip


def test_the_shapes_below_are_cut_in_every_way() -> None:
    """What `b200_gemm_plan` says of them on this device: (columns of a tile, CTAs per split tile, columns of the last round's parts)."""
    torch.cuda.current_device()
    plan, found = (ctypes.c_int32 * 3)(), set()
    for shape in PLANS:
        assert _lib.library().b200_gemm_plan(*shape, 0, None, plan) == _lib.OK
        found.add(tuple(plan))
    splits = {(64, s, 0) for s in (1, 2, 3, 4, 6, 8)}
    pairs = {(bn, 0, 0) for bn in (64, 128, 192, 256)}
    assert found == splits | pairs | {(256, 0, 64), (256, 0, 128)}


@pytest.mark.parametrize(("m", "n", "k"), PLANS)
def test_every_cut_of_a_product(m: int, n: int, k: int) -> None:
    x, w, bias, scale, res = (t.cuda() for t in operands(m, n, k, torch.bfloat16, seed=m + k))
    out = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    check(ff.gemm(x, w, bias, scale=scale, res=res, act=ff.ACT_GELU, out=out), x, w, bias, scale, res, act=ff.ACT_GELU, what=f"[{m},{n},{k}]")


@pytest.mark.parametrize("shapes", [
    ((1051, 2696, 520), (1051, 2696, 72)),  # one item per pair of CTAs; more k blocks than stages, and fewer
    ((2309, 2824, 72), (3863, 2824, 200)),  # two and three
    ((3345, 2888, 72), (4640, 2888, 200)),  # the last ones parts of a tile, some with all columns behind n
])  # fmt: skip
def test_last_items_of_a_pair_of_ctas_with_the_next_kernel_behind(shapes: tuple[tuple[int, int, int], ...]) -> None:
    """Two products in turn, the next one's CTAs taking the SMs as soon as a pair has gone: every repeat has the bits of the first."""
    cases = [tuple(t.cuda() for t in operands(m, n, k, torch.float16, seed=m + k)) for m, n, k in shapes]
    outs = [[torch.full((m, n), float("nan"), dtype=torch.float16, device="cuda") for _ in range(20)] for m, n, _ in shapes]
    for i in range(20):
        for (x, w, bias, _, res), out in zip(cases, outs, strict=True):
            ff.gemm(x, w, bias, res=res if i % 2 else None, out=out[i])
    for (x, w, bias, _, res), out, shape in zip(cases, outs, shapes, strict=True):
        check(out[0], x, w, bias, what=f"{shape}")
        check(out[1], x, w, bias, None, res, what=f"{shape} with a residual")
        assert all(torch.equal(out[i], out[i % 2]) for i in range(20))


def test_row_strided_views_and_leading_dims() -> None:
    """x, res and out as 2-D views with a row stride (lda, lres, ldy) and x with leading batch dims."""
    gen = torch.Generator().manual_seed(5)
    big = torch.randn(200, 160, generator=gen).half().cuda()
    x = big[:, 8:80]  # [200, 72], row stride 160
    w = (torch.randn(48, 72, generator=gen) * 0.1).half().cuda()
    canvas = torch.full((200, 96), 7.0, dtype=torch.float16, device="cuda")
    out = canvas[:, 16:64]
    ff.gemm(x, w, out=out)
    check(out, x, w, what="strided")
    assert bool((canvas[:, :16] == 7.0).all()) and bool((canvas[:, 64:] == 7.0).all())  # nothing outside the view
    x3 = torch.randn(3, 50, 72, generator=gen).half().cuda()
    got = ff.gemm(x3, w)
    assert got.shape == (3, 50, 48)
    check(got.reshape(150, 48), x3.reshape(150, 72), w, what="leading dims")


def test_contract_violations_raise_before_launch() -> None:
    x = torch.zeros(16, 64, dtype=torch.float16, device="cuda")
    w = torch.zeros(32, 64, dtype=torch.float16, device="cuda")
    with pytest.raises(ValueError, match="weight"):
        ff.gemm(x, w.t())
    with pytest.raises(ValueError, match="multiples of 8"):
        ff.gemm(x[:, :60].contiguous(), w[:, :60].contiguous())
    with pytest.raises(ValueError, match="bias"):
        ff.gemm(x, w, torch.zeros(31, dtype=torch.float16, device="cuda"))
    with pytest.raises(ValueError, match="scale"):
        ff.gemm(x, w, scale=torch.zeros(32, dtype=torch.float16, device="cuda"))
    with pytest.raises(ValueError, match="act"):
        ff.gemm(x, w, act=3)
    with pytest.raises(ValueError, match="requires grad"):
        ff.gemm(x.clone().requires_grad_(), w)
