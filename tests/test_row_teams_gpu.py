"""The streaming passes with a CTA to a row, at the lengths where their accesses, chunks and row groups end.

Held to torch with the same single operations in fp32, bit for bit; the fp32 row sums, whose order torch does not
have, to the oracle's order (scores) and to fp64 within n * 2^-24 of a sum of n non-negative terms (squares).
"""

from __future__ import annotations

import pytest
import torch

from dionw_b200 import _native as native
from oracle import dion_oracle as oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
# cols on both sides of every line at which the launch changes, of chunks of 1024, and of 16-, 8- and 4-byte accesses
COLS = [299, 300, 302, 767, 768, 1022, 1024, 1025, 1028, 2047, 2048, 2052, 2558, 2560, 4095, 4096, 4097, 4100, 5002]


def _gen(cols: int) -> torch.Generator:
    return torch.Generator(device=DEV).manual_seed(cols)


@pytest.mark.parametrize("cols", COLS)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_accumulate(cols: int, dtype: torch.dtype) -> None:
    gen = _gen(cols)
    rows = [3, 1, 6]   # groups of two and four rows end in the middle of the second and third tensor
    grads = [torch.randn(r, cols, device=DEV, generator=gen).to(dtype) for r in rows]
    start = torch.randn(1, sum(rows), cols, device=DEV, generator=gen)
    total = start[0] + torch.cat(grads).float()

    def squares_close(sums: torch.Tensor, of: torch.Tensor) -> bool:
        exact = of.double().square().sum(-1)
        return bool(((sums.flatten().double() - exact).abs() <= 2 * cols * 2.0**-24 * exact).all())

    momentum = start.clone()
    scores, sumsq = (torch.full((1, sum(rows)), 7.0, device=DEV) for _ in range(2))
    native.accumulate_row_l1_run(grads, rows, momentum, scores, sumsq, cols)
    assert torch.equal(momentum[0], total)
    assert torch.equal(scores.cpu(), oracle.row_scores(total.cpu()).view(1, -1))
    assert squares_close(sumsq, total)
    for nesterov in (False, True):
        momentum, u = start.clone(), torch.empty_like(start)
        native.accumulate_copy_decay_run(grads, rows, momentum, u, sumsq, cols, 0.95, nesterov)
        assert torch.equal(momentum[0], total * 0.95)
        assert torch.equal(u[0], torch.cat(grads).float() + total * 0.95 if nesterov else total)
        assert squares_close(sumsq, u[0])


@pytest.mark.parametrize("cols", [768, 1000, 1024, 1536, 2048, 4096])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_accumulate_gradients_off_a_boundary(cols: int, dtype: torch.dtype) -> None:
    """Gradients that start one element behind a 16-byte boundary, in rows that 4 divides: no wide access is allowed."""
    gen = _gen(cols)
    rows = [2, 5]
    grads = [torch.randn(r * cols + 1, device=DEV, generator=gen).to(dtype)[1:].view(r, cols) for r in rows]
    start = torch.randn(1, sum(rows), cols, device=DEV, generator=gen)
    total = start[0] + torch.cat(grads).float()
    momentum, u = start.clone(), torch.empty_like(start)
    scores, sumsq = (torch.full((1, sum(rows)), 7.0, device=DEV) for _ in range(2))
    native.accumulate_copy_decay_run(grads, rows, momentum, u, sumsq, cols, 0.95, False)
    assert torch.equal(momentum[0], total * 0.95) and torch.equal(u[0], total)
    momentum = start.clone()
    native.accumulate_row_l1_run(grads, rows, momentum, scores, sumsq, cols)
    assert torch.equal(momentum[0], total) and torch.equal(scores.cpu(), oracle.row_scores(total.cpu()).view(1, -1))


@pytest.mark.parametrize("cols", COLS)
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("selecting", [False, True])
def test_pack(cols: int, dtype: torch.dtype, selecting: bool) -> None:
    gen = _gen(cols)
    blocks, rows, k, ld = 2, 9, 5 if selecting else 9, (cols + 7) // 8 * 8
    source = torch.randn(blocks, rows, cols, device=DEV, generator=gen)
    index = torch.stack([torch.randperm(rows, device=DEV, generator=gen)[:k].sort().values for _ in range(blocks)]).int()
    frob = torch.tensor([3.7, 11.0], device=DEV)
    x = torch.full((blocks, k, ld), 77.0, dtype=dtype, device=DEV)
    after = source.clone()
    native.pack_rows(after, index if selecting else None, frob, k, x, decay=0.95, decay_rows=selecting, eps=1e-3, norm_scale=1.02)
    chosen = torch.stack([s[i.long()] for s, i in zip(source, index)]) if selecting else source
    if dtype is torch.bfloat16:
        denom = (frob.bfloat16() * 1.02 + 1e-3)[:, None, None]   # rounded after each step, as torch rounds
        want = chosen.bfloat16() / denom
    else:
        want = (chosen / (frob + 1e-3)[:, None, None]).half()
    assert torch.equal(x[..., :cols], want) and bool((x[..., cols:] == 0).all())
    if selecting:
        for s, i in zip(source, index):
            s[i.long()] *= 0.95
    assert torch.equal(after, source)


@pytest.mark.parametrize("per_sm", [6, 7, 8, 9])
@pytest.mark.parametrize("cols", [1001, 1024, 1026, 2048])
def test_accumulate_a_wave_of_rows(per_sm: int, cols: int) -> None:
    """About as many rows as a wave of warps takes, where the launch changes with their number."""
    rows = per_sm * torch.cuda.get_device_properties(DEV).multi_processor_count + 1 - (per_sm == 8)
    gen = _gen(cols)
    grad, start = torch.randn(rows, cols, device=DEV, generator=gen), torch.randn(1, rows, cols, device=DEV, generator=gen)
    total = start[0] + grad
    scores, sumsq = (torch.full((1, rows), 7.0, device=DEV) for _ in range(2))
    momentum, u = start.clone(), torch.empty_like(start)
    native.accumulate_copy_decay_run([grad], [rows], momentum, u, sumsq, cols, 0.95, False)
    assert torch.equal(momentum[0], total * 0.95) and torch.equal(u[0], total)
    momentum = start.clone()
    native.accumulate_row_l1_run([grad], [rows], momentum, scores, sumsq, cols)
    assert torch.equal(momentum[0], total) and torch.equal(scores.cpu(), oracle.row_scores(total.cpu()).view(1, -1))


# whole blocks on both sides of each line at which the launch changes with the number of rows
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows, cols", [(4096, 1025), (4097, 1025), (4097, 1602), (8192, 1601), (8193, 1601), (8193, 2561), (8192, 2560), (8193, 2560),
                                        (8193, 3072), (8193, 4096), (16385, 4096), (16385, 6144)])
def test_pack_many_whole_blocks(rows: int, cols: int, dtype: torch.dtype) -> None:
    source = torch.randn(1, rows, cols, device=DEV, generator=_gen(cols))
    frob = torch.tensor([5.0], device=DEV)
    x = torch.full((1, rows, (cols + 7) // 8 * 8), 77.0, dtype=dtype, device=DEV)
    native.pack_rows(source, None, frob, rows, x, decay=1.0, decay_rows=False, eps=1e-3, norm_scale=1.02)
    want = (source / (frob + 1e-3)).half() if dtype is torch.float16 else source.bfloat16() / (frob.bfloat16() * 1.02 + 1e-3)
    assert torch.equal(x[..., :cols], want) and bool((x[..., cols:] == 0).all())


@pytest.mark.parametrize("cols", COLS)
@pytest.mark.parametrize("selecting", [False, True])
@pytest.mark.parametrize("decay", [None, 0.9])
def test_apply(cols: int, selecting: bool, decay: float | None) -> None:
    gen = _gen(cols)
    rows, counts, ld = 7, [1, 2], (cols + 7) // 8 * 8
    blocks, k = sum(counts), 3 if selecting else 7
    weights = [torch.randn(n * rows, cols, device=DEV, generator=gen) for n in counts]
    update = torch.randn(blocks, k, ld, device=DEV, generator=gen).bfloat16()
    denom, scale = torch.rand(blocks * k, device=DEV, generator=gen) + 0.5, torch.rand(blocks, device=DEV, generator=gen)
    rowmap = torch.full((blocks, rows), -1, dtype=torch.int32, device=DEV)
    chosen = [torch.randperm(rows, device=DEV, generator=gen)[:k].sort().values for _ in range(blocks)]
    if selecting:
        for m, c in zip(rowmap, chosen):
            m[c] = torch.arange(k, dtype=torch.int32, device=DEV)
    else:
        chosen = [torch.arange(rows, device=DEV)] * blocks
    want = torch.cat(weights).view(blocks, rows, cols).clone()
    if decay is not None:
        want *= decay
    for b in range(blocks):
        want[b, chosen[b]] += update[b, :, :cols].float() / denom[b * k:(b + 1) * k, None] * scale[b]
    first = [0, counts[0]]
    native.apply_round(weights, [n * rows for n in counts], [update[b].data_ptr() for b in first],
                       [rowmap[b].data_ptr() for b in first] if selecting else None,
                       [denom[b * k:].data_ptr() for b in first], [scale[b:].data_ptr() for b in first], ldo=ld, rows=rows, k=k,
                       cols=cols, decay_factor=decay or 1.0, has_decay=decay is not None, decay_device=None, cta_warps=0, decay_job=None)
    assert torch.equal(torch.cat(weights).view(blocks, rows, cols), want)


# sparse updates of many rows, on both sides of each line at which the launch changes with their number and share
@pytest.mark.parametrize("rows, k, cols, decay", [
    (2000, 40, 302, None), (6000, 400, 302, None), (6000, 500, 302, None), (20000, 5290, 302, None), (20000, 5310, 302, None),
    (4000, 10, 302, 0.9), (5200, 400, 302, 0.9), (12000, 3950, 302, 0.9), (12000, 3975, 302, 0.9), (16384, 1, 2560, None),
    (16500, 20, 2560, None), (16500, 50, 2560, None), (32768, 6553, 2560, None), (32768, 6554, 2560, None), (32768, 1, 2560, 0.9),
    (8192, 8192, 2560, 0.9), (8193, 8193, 2560, 0.9), (8193, 8193, 2944, 0.9)])
def test_apply_few_of_many_rows(rows: int, k: int, cols: int, decay: float | None) -> None:
    gen = _gen(cols)
    weight = torch.randn(rows, cols, device=DEV, generator=gen)
    update = torch.randn(1, k, (cols + 7) // 8 * 8, device=DEV, generator=gen).bfloat16()
    denom, scale = torch.rand(k, device=DEV, generator=gen) + 0.5, torch.rand(1, device=DEV, generator=gen)
    chosen = torch.randperm(rows, device=DEV, generator=gen)[:k].sort().values
    rowmap = torch.full((1, rows), -1, dtype=torch.int32, device=DEV)
    rowmap[0, chosen] = torch.arange(k, dtype=torch.int32, device=DEV)
    want = weight * decay if decay is not None else weight.clone()
    want[chosen] += update[0, :, :cols].float() / denom[:, None] * scale
    native.apply_run([weight], [rows], update, rowmap, denom, scale, rows=rows, k=k, cols=cols, decay_factor=decay or 1.0,
                     has_decay=decay is not None)
    assert torch.equal(weight, want)


def test_selections_and_scales_of_several_runs_in_one_launch() -> None:
    """Runs of one CTA to a block beside runs of eight: each gets what it gets alone, bit for bit."""
    gen = _gen(1)
    shapes = [(3, 300, 75), (1, 9000, 2000), (2, 1025, 1025), (5, 64, 1), (1, 4000, 3999), (2, 2048, 512)]   # blocks, rows, k
    assert len(shapes) == native.NS_GROUP_MAX

    def selection(scores: torch.Tensor, k: int) -> tuple:
        index = torch.full((scores.shape[0], k), -7, dtype=torch.int32, device=DEV)
        rowmap = torch.full(scores.shape, -7, dtype=torch.int32, device=DEV)
        return scores, scores.square(), k, index, rowmap, torch.full((scores.shape[0],), 7.0, device=DEV)

    scores = [torch.rand(blocks, rows, device=DEV, generator=gen) for blocks, rows, _ in shapes]
    together = [selection(s, k) for s, (_, _, k) in zip(scores, shapes)]
    native.select_rows_group(together)
    for s, (_, _, k), run in zip(scores, shapes, together):
        alone = selection(s, k)
        native.select_rows(*alone)
        assert all(torch.equal(run[i], alone[i]) for i in (3, 4, 5))

    def scales(i: int) -> dict:
        blocks, rows, k = shapes[i]
        sums = torch.rand(blocks * k, 4, device=DEV, generator=_gen(i)) + 0.1
        return {"s": sums, "parts": 4, "variance": torch.rand(blocks, rows, device=DEV, generator=_gen(i + 10)),
                "index": None if i == 2 else together[i][3], "blocks": blocks, "rows": rows, "k": k, "cols": 500, "weight": 0.05 * (i + 1),
                "step": -0.01 * (i + 1), "step_device": torch.tensor([0.5], device=DEV) if i == 1 else None, "normalize": i != 4,
                "denom": torch.zeros(blocks * k, device=DEV), "scale": torch.zeros(blocks, device=DEV)}

    grouped = [scales(i) for i in range(len(shapes))]
    native.normuon_rows_group(grouped, 1e-8)
    for i, run in enumerate(grouped):
        alone = scales(i)
        native.normuon_rows(**alone, eps=1e-8)
        assert all(torch.equal(run[key], alone[key]) for key in ("variance", "denom", "scale"))
    with pytest.raises(ValueError, match="1 to 6"):
        native.select_rows_group(together + together[:1])


def test_many_narrow_blocks_beside_a_wide_one_have_their_own_launch() -> None:
    """Blocks of one CTA would otherwise each take the eight of the widest run; same values either way."""
    gen = _gen(2)
    shapes = [(300, 128, 32), (1, 9000, 2000), (2, 4000, 1024), (500, 100, 100)]   # blocks, rows, k

    def runs() -> tuple[list, list]:
        selections, scales = [], []
        for i, (blocks, rows, k) in enumerate(shapes):
            scores = torch.rand(blocks, rows, device=DEV, generator=_gen(i))
            index = torch.full((blocks, k), -7, dtype=torch.int32, device=DEV)
            selections.append((scores, scores.square(), k, index, torch.full((blocks, rows), -7, dtype=torch.int32, device=DEV),
                               torch.full((blocks,), 7.0, device=DEV)))
            scales.append({"s": torch.rand(blocks * k, 2, device=DEV, generator=_gen(i)) + 0.1, "parts": 2,
                           "variance": torch.rand(blocks, rows, device=DEV, generator=_gen(i)), "index": index, "blocks": blocks, "rows": rows,
                           "k": k, "cols": 500, "weight": 0.05, "step": -0.01, "step_device": None, "normalize": True,
                           "denom": torch.zeros(blocks * k, device=DEV), "scale": torch.zeros(blocks, device=DEV)})
        return selections, scales

    (together, grouped), (alone, single) = runs(), runs()
    before = native.launch_count()
    native.select_rows_group(together)
    native.normuon_rows_group(grouped, 1e-8)
    assert native.launch_count() - before == 2 + 2   # the two wide runs, the two narrow ones
    for run, own, group, lone in zip(together, alone, grouped, single):
        native.select_rows(*own)
        native.normuon_rows(**lone, eps=1e-8)
        assert all(torch.equal(run[i], own[i]) for i in (3, 4, 5))
        assert all(torch.equal(group[key], lone[key]) for key in ("variance", "denom", "scale"))
    before = native.launch_count()
    native.select_rows_group(together[1:3])
    assert native.launch_count() - before == 1
