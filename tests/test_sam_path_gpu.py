"""SAM's attention with the decomposed relative-position term, side by side with the path the reference runs.

For SAM the reference's kernels mode does not call `flash64_*`: it folds the bias into the dot product by widening
q and k ("augmented", `src/fastforks/promptable_segmentation/models/sam/fast.py:92-113`: `q' = [q * scale | rel_h |
rel_w | 0]`, `k' = [k | onehot(kh) | onehot(kw) | 0]`, `v' = [v | 0]`, head dim 96 for 14 x 14 windows and 192 for the
64 x 64 grid) and calls `F.scaled_dot_product_attention(..., scale=1.0)[..., :64]` (`fused.py:80-86`). This file
restates that construction (test infrastructure: torch ops only) and

  * checks this library's `rel=(rel_h, rel_w)` call against it on the same packed qkv and tables (same operands, two
    different routes to the same logits: the bar is the path's op-level tolerance), and
  * times both, each including the two einsums that produce `rel_h`, `rel_w` from q and the tables (both routes
    need them) and, for the reference's route, the three concatenations it needs on top; and this library once more
    with its own producer kernel (`b200_sam_rel_terms`) in place of the einsums, which is also checked against the
    oracle on its own.

Speed is reported (JSON to $B200_SAM_SIDE_BY_SIDE when set), not gated.
"""

from __future__ import annotations

import json
import os

import pytest
import torch

import fastforks_b200 as ff
from conftest import assert_close

pytestmark = pytest.mark.gpu

HEADS, DIM = 12, 64
SHAPES = {"sam-vit-b windows [25,12,196,64]": (25, 14), "sam-vit-b global [1,12,4096,64]": (1, 64)}


def onehot_keys(side: int) -> torch.Tensor:
    """`[side * side, 2 * side]`: key (a, c) has a one in column a and in column side + c (fast.py:85-89)."""
    eye = torch.eye(side, device="cuda", dtype=torch.float16)
    return torch.cat([eye.repeat_interleave(side, 0), eye.repeat(side, 1)], 1)


def rel_terms(qkv: torch.Tensor, rh: torch.Tensor, rw: torch.Tensor, side: int) -> tuple[torch.Tensor, torch.Tensor]:
    """`rel_h`, `rel_w` `[B, heads, N, side]` from the unscaled q and the tables `[side, side, 64]` (fast.py:104-106)."""
    b, n = qkv.shape[:2]
    r_q = qkv[:, :, 0].reshape(b, side, side, HEADS, DIM)
    rel_h = torch.einsum("bhwnc,hkc->bnhwk", r_q, rh).reshape(b, HEADS, n, side)
    rel_w = torch.einsum("bhwnc,wkc->bnhwk", r_q, rw).reshape(b, HEADS, n, side)
    return rel_h, rel_w


def reference_route(qkv: torch.Tensor, rh: torch.Tensor, rw: torch.Tensor, onehot: torch.Tensor, side: int) -> torch.Tensor:
    """Widened operands + SDPA with scale 1, sliced back to 64 columns: `[B, heads, N, 64]` (fast.py:92-113, 128-135)."""
    b, n = qkv.shape[:2]
    q, k, v = qkv.unbind(2)
    rel_h, rel_w = rel_terms(qkv, rh, rw, side)
    pad = -(DIM + 2 * side) % 8
    qt = q.transpose(1, 2)
    zeros = qt.new_zeros(b, HEADS, n, pad)
    qa = torch.cat([qt * DIM**-0.5, rel_h, rel_w, zeros], -1)
    ka = torch.cat([k.transpose(1, 2), onehot.expand(b, HEADS, n, 2 * side), zeros], -1)
    va = torch.cat([v.transpose(1, 2), qt.new_zeros(b, HEADS, n, 2 * side + pad)], -1)
    return torch.nn.functional.scaled_dot_product_attention(qa, ka, va, scale=1.0)[..., :DIM]


def this_library(qkv: torch.Tensor, rh: torch.Tensor, rw: torch.Tensor, side: int) -> torch.Tensor:
    """The same attention through `rel=`: q, k, v stay 64 wide views of the packed tensor. `[B, N, heads, 64]`."""
    q, k, v = qkv.unbind(2)
    return ff.attention(q, k, v, scale=DIM**-0.5, layout="bnhd", rel=rel_terms(qkv, rh, rw, side))


def this_library_with_producer(qkv: torch.Tensor, pos_h: torch.Tensor, pos_w: torch.Tensor, side: int) -> torch.Tensor:
    """The same with `rel_h`, `rel_w` from this library's producer kernel, which reads q in place and the module's
    `[2 * side - 1, 64]` parameters instead of gathered tables."""
    q, k, v = qkv.unbind(2)
    return ff.attention(q, k, v, scale=DIM**-0.5, layout="bnhd", rel=ff.sam_rel_terms(q, pos_h, pos_w, side))


def gathered(pos: torch.Tensor, side: int) -> torch.Tensor:
    """`[side, side, 64]` table of a `[2 * side - 1, 64]` parameter (upstream `get_rel_pos`, equal sizes)."""
    idx = torch.arange(side, device=pos.device)
    return pos[(idx[:, None] - idx[None, :]) + (side - 1)]


@pytest.mark.parametrize(("b", "side", "dtype"), [(25, 14, torch.float16), (1, 64, torch.float16), (3, 14, torch.bfloat16), (2, 8, torch.bfloat16), (1, 64, torch.bfloat16)])
def test_producer_kernel_matches_the_oracle(b: int, side: int, dtype: torch.dtype) -> None:
    """`b200_sam_rel_terms` against the oracle's restatement of the two einsums of `add_decomposed_rel_pos`
    (oracle/attention_oracle.py: decomposed_terms) on the rounded operands; results are rounded to 16 bits once."""
    from oracle import attention_oracle as ao

    gen = torch.Generator().manual_seed(side + b)
    qkv = torch.randn(b, side * side, 3, HEADS, DIM, generator=gen).to(dtype).cuda()
    pos_h, pos_w = ((torch.randn(2 * side - 1, DIM, generator=gen) * 0.1).to(dtype).cuda() for _ in range(2))
    rel_h, rel_w = ff.sam_rel_terms(qkv[:, :, 0], pos_h, pos_w, side)
    q = qkv[:, :, 0].float().cpu().numpy().transpose(0, 2, 1, 3)
    want_h, want_w = ao.decomposed_terms(q, pos_h.float().cpu().numpy(), pos_w.float().cpu().numpy(), (side, side))
    assert_close(rel_h.float().cpu().numpy(), want_h, unit_scale=False, what=f"rel_h side {side} {dtype}")
    assert_close(rel_w.float().cpu().numpy(), want_w, unit_scale=False, what=f"rel_w side {side} {dtype}")


@pytest.mark.parametrize(("b", "side", "heads"), [(1, 2, 1), (2, 6, 3), (1, 10, 17), (1, 16, 16), (1, 22, 24), (3, 32, 12), (1, 40, 5), (1, 48, 33), (2, 50, 12), (1, 62, 7),
                                                  (1, 64, 1), (1, 64, 17), (3, 56, 2), (70, 14, 2)])  # fmt: skip
def test_producer_kernel_at_every_tile_count(b: int, side: int, heads: int) -> None:
    """Grid sides for each number of eight-column tiles, head counts around the sixteen rows of one product, and a second
    table whose address is only 4-byte aligned (read word by word)."""
    from oracle import attention_oracle as ao

    gen = torch.Generator().manual_seed(side * heads)
    qkv = torch.randn(b, side * side, 3, heads, DIM, generator=gen).half().cuda()
    values = (torch.randn(2, 2 * side - 1, DIM, generator=gen) * 0.1).half().cuda()
    room = torch.empty(2 + values[1].numel(), dtype=torch.float16, device="cuda")
    both = [values[0], room[2:].view_as(values[1]).copy_(values[1])]
    rel_h, rel_w = ff.sam_rel_terms(qkv[:, :, 0], both[0], both[1], side)
    want_h, want_w = ao.decomposed_terms(qkv[:, :, 0].float().cpu().numpy().transpose(0, 2, 1, 3), *(t.float().cpu().numpy() for t in both), (side, side))
    assert_close(rel_h.float().cpu().numpy(), want_h, unit_scale=False, what=f"rel_h side {side}")
    assert_close(rel_w.float().cpu().numpy(), want_w, unit_scale=False, what=f"rel_w side {side}")
    assert ff.device_status() == 0


@pytest.mark.parametrize(("b", "side", "heads"), [(2, 40, 2), (1, 40, 5), (2, 48, 3), (1, 56, 12), (1, 64, 16), (1, 64, 33)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_producer_kernel_by_lines(b: int, side: int, heads: int, dtype: torch.dtype) -> None:
    """Aligned tables at the sides a line at a time is computed for: one tile of rows and less, ragged last tiles, more tiles than
    tensor memory holds at once, and numbers of columns that are no multiple of the product's sixteen."""
    from oracle import attention_oracle as ao

    gen = torch.Generator().manual_seed(side + heads)
    qkv = torch.randn(b, side * side, 3, heads, DIM, generator=gen).to(dtype).cuda()
    pos_h, pos_w = ((torch.randn(2 * side - 1, DIM, generator=gen) * 0.1).to(dtype).cuda() for _ in range(2))
    rel_h, rel_w = ff.sam_rel_terms(qkv[:, :, 1], pos_h, pos_w, side)
    want_h, want_w = ao.decomposed_terms(qkv[:, :, 1].float().cpu().numpy().transpose(0, 2, 1, 3), pos_h.float().cpu().numpy(), pos_w.float().cpu().numpy(), (side, side))
    assert ff.device_status() == 0
    assert_close(rel_h.float().cpu().numpy(), want_h, unit_scale=False, what=f"rel_h side {side}")
    assert_close(rel_w.float().cpu().numpy(), want_w, unit_scale=False, what=f"rel_w side {side}")


@pytest.mark.parametrize(("b", "side", "heads"), [(1, 40, 12), (1, 48, 5), (2, 56, 3), (1, 64, 12), (1, 64, 17)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_producer_kernels_give_the_same_bits(b: int, side: int, heads: int, dtype: torch.dtype) -> None:
    """The same tables on 16 bytes (by lines) and on 4 (by tokens): both add a term's 64 products in the same order."""
    gen = torch.Generator(device="cuda").manual_seed(side + heads)
    q = torch.randn(b, side * side, heads, DIM, generator=gen, device="cuda").to(dtype)
    pos = (torch.randn(2, 2 * side - 1, DIM, generator=gen, device="cuda") * 0.1).to(dtype)
    apart = torch.empty(2, 2 + pos[0].numel(), dtype=dtype, device="cuda")[:, 2:].unflatten(1, pos.shape[1:]).copy_(pos)
    assert [t.data_ptr() % 16 for t in pos] == [0, 0]
    assert [t.data_ptr() % 16 != 0 for t in apart] == [True, True]
    for by_lines, by_tokens in zip(ff.sam_rel_terms(q, *pos, side), ff.sam_rel_terms(q, *apart, side), strict=True):
        assert torch.equal(by_lines, by_tokens)


@pytest.mark.parametrize(("b", "side", "heads"), [(80, 8, 3), (70, 14, 17), (54, 20, 2), (31, 26, 1), (16, 32, 3), (8, 40, 2), (4, 40, 3), (3, 64, 1), (3, 64, 12), (2, 64, 16), (2, 64, 17)])
def test_producer_gives_an_image_the_same_bits_alone_and_in_a_batch(b: int, side: int, heads: int) -> None:
    """One image goes by tokens or by lines, as many tiles of rows at a time as there are; the batch by rows, by lines, or by lines with
    fewer tiles at a time."""
    gen = torch.Generator(device="cuda").manual_seed(side + heads)
    q = torch.randn(b, side * side, heads, DIM, generator=gen, device="cuda").half()
    pos = (torch.randn(2, 2 * side - 1, DIM, generator=gen, device="cuda") * 0.1).half()
    together = ff.sam_rel_terms(q, *pos, side)
    for i in {0, b // 2, b - 1}:
        for whole, alone in zip(together, ff.sam_rel_terms(q[i : i + 1], *pos, side), strict=True):
            assert torch.equal(whole[i], alone[0])


@pytest.mark.parametrize(("b", "side", "heads"), [(1, 40, 2), (3, 40, 6), (2, 64, 4), (2, 64, 12), (1, 64, 33)])
def test_producer_by_lines_with_kernels_close_behind(b: int, side: int, heads: int) -> None:
    """Kernels that allocate tensor memory in their set-up, each started while the one in front drains: lines of one to eight tiles and
    more, then a product cut along k, one in pairs, and attention. Every round gives what the first one gave."""
    gen = torch.Generator(device="cuda").manual_seed(side * heads)
    q, k, v = torch.randn(b, side * side, 3, heads, DIM, generator=gen, device="cuda").half().unbind(2)
    pos_h, pos_w = ((torch.randn(2 * side - 1, DIM, generator=gen, device="cuda") * 0.1).half() for _ in range(2))
    small, wide, w = (torch.randn(m, 512, generator=gen, device="cuda").half() for m in (100, 4000, 1024))
    first = None
    for _ in range(12):
        rel = ff.sam_rel_terms(q, pos_h, pos_w, side)
        out = [*rel, ff.gemm(small, w)]
        out += [*ff.sam_rel_terms(k, pos_h, pos_w, side), ff.gemm(wide, w)]
        out += [*ff.sam_rel_terms(v, pos_h, pos_w, side), ff.attention(q, k, v, scale=DIM**-0.5, layout="bnhd", rel=rel)]
        first = first or out
        assert all(torch.equal(x, y) for x, y in zip(out, first, strict=True))
    assert ff.device_status() == 0
    for got, x in ((first[2], small), (first[5], wide)):
        assert_close(got.float().cpu().numpy(), (x.float() @ w.float().T).cpu().numpy(), unit_scale=False, what=f"product behind [{b},{side},{heads}]")


def test_producer_kernel_rejects_what_it_cannot_take() -> None:
    q = torch.zeros(1, 25, 2, 64, dtype=torch.float16, device="cuda")
    pos = torch.zeros(9, 64, dtype=torch.float16, device="cuda")
    with pytest.raises(ValueError, match="grid"):
        ff.sam_rel_terms(q, pos, pos, 4)
    with pytest.raises(ValueError, match="even"):
        ff.sam_rel_terms(q, pos, pos, 5)
    with pytest.raises(ValueError, match="rel_pos_h"):
        ff.sam_rel_terms(q[:, :16], pos, pos, 4)


def operands(b: int, side: int, seed: int) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    gen = torch.Generator().manual_seed(seed)
    qkv = torch.randn(b, side * side, 3, HEADS, DIM, generator=gen).half().cuda()
    rh, rw = ((torch.randn(side, side, DIM, generator=gen) * 0.1).half().cuda() for _ in range(2))
    return qkv, rh, rw


def parameters(side: int, seed: int) -> tuple[torch.Tensor, torch.Tensor]:
    gen = torch.Generator().manual_seed(1000 + seed)
    return tuple((torch.randn(2 * side - 1, DIM, generator=gen) * 0.1).half().cuda() for _ in range(2))


@pytest.mark.parametrize("name", list(SHAPES))
def test_same_result_as_the_reference_route(name: str) -> None:
    b, side = SHAPES[name]
    qkv, _, _ = operands(b, side, seed=side)
    pos_h, pos_w = parameters(side, side)
    rh, rw = gathered(pos_h, side), gathered(pos_w, side)
    theirs = reference_route(qkv, rh, rw, onehot_keys(side), side).transpose(1, 2)
    ours = this_library(qkv, rh, rw, side)
    assert_close(ours.float().cpu().numpy(), theirs.float().cpu().numpy(), unit_scale=True, what=name)
    fused = this_library_with_producer(qkv, pos_h, pos_w, side)
    assert_close(fused.float().cpu().numpy(), theirs.float().cpu().numpy(), unit_scale=True, what=name + " (producer kernel)")
    assert ff.device_status() == 0


def _time_us(fn, reps: int = 20) -> float:  # noqa: ANN001
    for _ in range(5):
        fn()
    torch.cuda.synchronize()
    best = float("inf")
    for _ in range(5):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(reps):
            fn()
        e1.record()
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1) / reps * 1e3)
    return best


def test_times_side_by_side_with_the_reference_route() -> None:
    rows = {}
    for name, (b, side) in SHAPES.items():
        sets = [operands(b, side, seed=i) for i in range(8)]  # 8 x 19-30 MB of qkv: rotating, larger than L2 together
        onehot = onehot_keys(side)
        state = {"i": 0}

        def nxt() -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
            state["i"] = (state["i"] + 1) % len(sets)
            return sets[state["i"]]

        pos_h, pos_w = parameters(side, 0)
        rel_only = _time_us(lambda: rel_terms(*nxt(), side))
        producer_only = _time_us(lambda: ff.sam_rel_terms(nxt()[0][:, :, 0], pos_h, pos_w, side))
        ours = _time_us(lambda: this_library(*nxt(), side))
        ours_producer = _time_us(lambda: this_library_with_producer(nxt()[0], pos_h, pos_w, side))
        theirs = _time_us(lambda: reference_route(*nxt(), onehot, side))
        rows[name] = {"rel_einsums_us": rel_only, "producer_kernel_us": producer_only, "this_library_with_einsums_us": ours,
                      "this_library_with_producer_kernel_us": ours_producer,
                      "reference_augmented_sdpa_with_einsums_us": theirs, "speedup": theirs / ours_producer}  # fmt: skip
        print(name, json.dumps(rows[name]))
    assert all(r["this_library_with_einsums_us"] > 0 for r in rows.values())
    assert ff.device_status() == 0
    path = os.environ.get("B200_SAM_SIDE_BY_SIDE")
    if path:
        with open(path, "w") as f:
            json.dump(rows, f, indent=1)
