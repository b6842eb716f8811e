"""The products' epilogue, the tall iteration and the normalising pack at the sizes where they can go wrong.

Products are held to the fp64 product of the same 2-byte operands.  One rounding of the result to fp16
(2^-11 relative) or bf16 (2^-8) and fp32 accumulation of at most 600 terms (below 600 * 2^-24 of the sum
of magnitudes) bound the difference.
"""

from __future__ import annotations

import pytest
import torch

from dionw_b200 import _native as native

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SENTINEL = 77.0


def _padded(n: int) -> int:
    return (n + 7) // 8 * 8


def _operand(gen: torch.Generator, blocks: int, rows: int, cols: int, dtype: torch.dtype) -> torch.Tensor:
    x = torch.zeros(blocks, rows, _padded(cols), dtype=dtype)
    x[..., :cols] = (torch.randn(blocks, rows, cols, generator=gen) * 0.1).to(dtype)
    return x.to(DEV)


def _close(got: torch.Tensor, want: torch.Tensor, magnitude: torch.Tensor, dtype: torch.dtype) -> None:
    rounding = 2.0**-11 if dtype is torch.float16 else 2.0**-8
    bound = rounding * want.abs() * 1.01 + 600 * 2.0**-24 * magnitude + 1e-7
    assert bool(((got.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("m", [1, 8, 31, 33, 64, 127, 130, 256, 257, 517])
def test_symmetric_products_at_every_edge(m: int, dtype: torch.dtype) -> None:
    gen = torch.Generator().manual_seed(m)
    blocks, k = 2, 45 + m
    a = _operand(gen, blocks, m, k, dtype)
    a64 = a[..., :k].double()
    want = a64 @ a64.mT
    size = a64.abs() @ a64.mT.abs()
    out = torch.full((blocks, m, _padded(m)), SENTINEL, dtype=dtype, device=DEV)
    out2 = out.clone()
    native.symmetric_product(a[..., :k], out[..., :m])
    _close(out[..., :m], want, size, dtype)
    assert torch.equal(out[..., :m], out[..., :m].mT) and bool((out[..., m:] == SENTINEL).all())
    # the polynomial form: Cin, two outputs, the second with a diagonal added to the rounded first
    g = out.clone()
    native.symmetric_product(g[..., :m], out[..., :m], cin=g[..., :m], alpha=0.5, beta=-1.25, out2=out2[..., :m], diag=2.5)
    g64 = g[..., :m].double()
    _close(out[..., :m], 0.5 * g64 @ g64 - 1.25 * g64, 0.5 * g64.abs() @ g64.abs() + 1.25 * g64.abs(), dtype)
    eye = torch.eye(m, device=DEV)
    assert torch.equal(out2[..., :m], (out[..., :m].float() + 2.5 * eye).to(dtype))
    # B != A, symmetric and commuting (a polynomial of A): exactly symmetric although only one triangle is computed
    z = out.clone()
    native.symmetric_product(g[..., :m], out[..., :m], b=z[..., :m], cin=g[..., :m], beta=1.5)
    z64 = z[..., :m].double()
    lower = torch.tril(g64 @ z64 + 1.5 * g64)
    _close(torch.tril(out[..., :m].double()), lower, g64.abs() @ z64.abs() + 1.5 * g64.abs(), dtype)
    assert torch.equal(out[..., :m], out[..., :m].mT) and bool((out[..., m:] == SENTINEL).all())


@pytest.mark.parametrize("m, n, k", [(1, 1, 1), (33, 70, 40), (130, 259, 65), (256, 256, 256), (300, 31, 129)])
@pytest.mark.parametrize("ld_extra", [0, 8, 3])
def test_general_products_leave_everything_outside_alone(m: int, n: int, k: int, ld_extra: int) -> None:
    """Also with an output whose rows are not 16-byte aligned (``ld_extra`` 3)."""
    gen = torch.Generator().manual_seed(n)
    a, b = _operand(gen, 2, m, k, torch.float16), _operand(gen, 2, k, n, torch.float16)
    c = torch.randn(2, m, _padded(n) + ld_extra, generator=gen).half().to(DEV)
    out = torch.full((2, m, _padded(n) + ld_extra), SENTINEL, dtype=torch.float16, device=DEV)
    native.batched_gemm(a[..., :k], b[..., :n], out[..., :n], b_is_nk=False, cin=c[..., :n], beta=-0.5)
    a64, b64, c64 = a[..., :k].double(), b[..., :n].double(), c[..., :n].double()
    _close(out[..., :n], a64 @ b64 - 0.5 * c64, a64.abs() @ b64.abs() + 0.5 * c64.abs(), torch.float16)
    assert bool((out[..., n:] == SENTINEL).all())


@pytest.mark.parametrize("kind", [native.NS_GRAM, native.NS_GRAM_FULL, native.NS_POLAR_EXPRESS, native.NS_KELLER])
@pytest.mark.parametrize("rows, cols", [(2, 1), (40, 33), (257, 256), (700, 65), (1531, 517)])
def test_tall_blocks_equal_the_iteration_of_their_transpose(rows: int, cols: int, kind: int) -> None:
    """Bit for bit: each element is the same dot product, accumulated in the same order."""
    gen = torch.Generator().manual_seed(rows)
    dtype = torch.float16 if kind in (native.NS_GRAM, native.NS_GRAM_FULL) else torch.bfloat16
    blocks = 3
    x = torch.randn(blocks, rows, cols, generator=gen)
    x = (x / x.norm(dim=(1, 2), keepdim=True)).to(dtype).to(DEV)
    tall = torch.zeros(blocks, rows, _padded(cols), dtype=dtype, device=DEV)
    tall[..., :cols] = x
    wide = torch.zeros(blocks, cols, _padded(rows), dtype=dtype, device=DEV)
    wide[..., :rows] = x.mT
    parts = native.newton_schulz_rowsq_parts(cols)
    rowsq = torch.full((blocks * rows, parts), SENTINEL, device=DEV)
    ws = torch.empty(native.newton_schulz_tall_workspace_bytes(blocks, rows, cols, kind), dtype=torch.uint8, device=DEV)
    native.newton_schulz_tall(tall, tall.view(torch.bfloat16), rows, cols, kind, ws, rowsq)
    ws = torch.empty(native.newton_schulz_workspace_bytes(blocks, cols, rows, kind), dtype=torch.uint8, device=DEV)
    native.newton_schulz(wide, wide.view(torch.bfloat16), cols, rows, kind, ws)
    got, want = tall.view(torch.bfloat16)[..., :cols], wide.view(torch.bfloat16)[..., :rows].mT
    assert torch.equal(got, want)
    # at most 128 fp32 additions per part of 128 columns (the parts are added in fp64 here): 2^-15 of a sum of squares
    exact = got.double().square().sum(-1).flatten()
    assert bool(((rowsq.double().sum(-1) - exact).abs() <= 2.0**-15 * exact + 1e-30).all())


@pytest.mark.parametrize("rows, cols", [(1, 1), (3, 1000), (40, 33), (257, 264), (64, 4100)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_normalize_pack_matches_the_fp32_form(rows: int, cols: int, dtype: torch.dtype) -> None:
    gen = torch.Generator().manual_seed(cols)
    src = (torch.randn(2, rows, cols, generator=gen) + 0.1).to(dtype)
    for out_dtype, scale in ((torch.float16, 1.0), (torch.bfloat16, 1.02)):
        x = torch.full((2, rows, _padded(cols)), SENTINEL, dtype=out_dtype, device=DEV)
        native.normalize_pack(src.to(DEV), x, eps=1e-8, norm_scale=scale)
        value = src.float() if out_dtype is torch.float16 else src.bfloat16().float()
        norm = value.double().square().sum((1, 2), keepdim=True).sqrt()
        # the norm's own last bits and, for bf16, three roundings of the divisor and one of the quotient
        bound = (2.0**-11 if out_dtype is torch.float16 else 4 * 2.0**-8) * 1.02
        want = value.double() / (norm * scale)
        assert bool(((x[..., :cols].double().cpu() - want).abs() <= bound * want.abs() + 2.0**-24).all())
        assert bool((x[..., cols:] == 0).all())


@pytest.mark.parametrize("blocks, rows, cols", [(1, 256, 1024), (6, 1531, 517), (16, 1024, 1024), (40, 65, 4000), (3, 1, 9)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_normalize_pack_has_the_bits_of_the_fp32_form(blocks: int, rows: int, cols: int, dtype: torch.dtype) -> None:
    """Bit for bit what the batch's fp32 copy gives, divided by torch's norm of that copy."""
    for seed in range(3):
        gen = torch.Generator(device=DEV).manual_seed(seed)
        src = torch.randn(blocks, rows, cols, device=DEV, generator=gen)
        if seed > 0:
            src /= torch.linalg.vector_norm(src, dim=(1, 2), keepdim=True)
        src = src.to(dtype)
        copy = src.float()
        for out_dtype, scale in ((torch.float16, 1.0), (torch.bfloat16, 1.02)):
            half = out_dtype is torch.float16
            norm = torch.linalg.vector_norm(copy, dim=(1, 2)) if half else copy.bfloat16().norm(dim=(1, 2)).float()
            x, want = (torch.empty(blocks, rows, _padded(cols), dtype=out_dtype, device=DEV) for _ in range(2))
            native.normalize_pack(src, x, eps=1e-8, norm_scale=scale)
            native.pack_rows(copy, None, norm, rows, want, decay=1.0, decay_rows=False, eps=1e-8, norm_scale=scale)
            assert torch.equal(x, want)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_the_library_takes_the_norms_of_a_caller_without_them(dtype: torch.dtype) -> None:
    """With a buffer for row sums the norms come from fp32 sums of 40 x 333 squares: 2^-12 at the most."""
    gen = torch.Generator(device=DEV).manual_seed(2)
    src = torch.randn(3, 40, 333, device=DEV, generator=gen).to(dtype)
    x = torch.empty(3, 40, 336, dtype=torch.float16, device=DEV)
    sums, frob = torch.empty(120, device=DEV), torch.empty(3, device=DEV)
    status = native.library().dionw_normalize_pack(
        src.data_ptr(), native.dtype_code(dtype), 3, 40, 333, 1e-8, 1.0, x.data_ptr(), native.F16, 336, sums.data_ptr(),
        frob.data_ptr(), torch.cuda.current_stream().cuda_stream)
    assert status == 0
    norm = src.double().square().sum((1, 2)).sqrt()
    assert bool(((frob.double() - norm).abs() <= 2.0**-12 * norm).all())
    want = torch.empty_like(x)
    native.pack_rows(src.float(), None, frob, 40, want, decay=1.0, decay_rows=False, eps=1e-8)
    assert torch.equal(x, want)


@pytest.mark.parametrize("kinds", [(native.NS_GRAM,), (native.NS_POLAR_EXPRESS, native.NS_KELLER)])
def test_a_group_of_batches_equals_its_members_alone(kinds: tuple[int, ...]) -> None:
    """One launch over wide, square and tall batches, of one tile and of many, against one launch each,
    bit for bit; repeated, because what could differ is the order in which tiles run."""
    shapes = [(3, 130, 300), (1, 1, 1), (2, 256, 256), (5, 700, 65), (1, 1030, 2100), (40, 64, 192)]
    assert len(shapes) == native.NS_GROUP_MAX
    gen = torch.Generator().manual_seed(5)
    dtype = torch.float16 if native.NS_GRAM in kinds else torch.bfloat16
    codes = [kinds[i % len(kinds)] for i in range(len(shapes))]
    sources, want, sums = [], [], []
    for (blocks, rows, cols), kind in zip(shapes, codes):
        x = torch.zeros(blocks, rows, _padded(cols), dtype=dtype)
        values = torch.randn(blocks, rows, cols, generator=gen)
        x[..., :cols] = (values / values.norm(dim=(1, 2), keepdim=True)).to(dtype)
        x = x.to(DEV)
        sources.append(x)
        alone = x.clone()
        rowsq = torch.empty(blocks * rows, native.newton_schulz_rowsq_parts(cols), device=DEV)
        tall = rows > cols
        need = (native.newton_schulz_tall_workspace_bytes if tall else native.newton_schulz_workspace_bytes)
        ws = torch.empty(need(blocks, rows, cols, kind), dtype=torch.uint8, device=DEV)
        run = native.newton_schulz_tall if tall else native.newton_schulz
        run(alone, alone.view(torch.bfloat16), rows, cols, kind, ws, rowsq)
        want.append(alone.view(torch.bfloat16)[..., :cols])
        sums.append(rowsq)
        stepwise, out = x.clone(), torch.empty_like(x).view(torch.bfloat16)
        run(stepwise, out, rows, cols, kind + native.NS_STEPWISE, ws)
        assert torch.equal(out[..., :cols], want[-1])
    ws = torch.empty(native.newton_schulz_group_workspace_bytes(shapes, codes), dtype=torch.uint8, device=DEV)
    for _ in range(5):
        ws.fill_(255)   # neither the counters nor the matrices may have to start at anything
        xs = [x.clone() for x in sources]
        rowsqs = [None if i == 2 else torch.full_like(s, SENTINEL) for i, s in enumerate(sums)]
        native.newton_schulz_group(xs, [x.view(torch.bfloat16) for x in xs], shapes, codes, ws, rowsqs)
        for i, (x, (_, _, cols)) in enumerate(zip(xs, shapes)):
            assert torch.equal(x.view(torch.bfloat16)[..., :cols], want[i])
            assert rowsqs[i] is None or torch.equal(rowsqs[i], sums[i])
    assert native.device_status() == 0
    with pytest.raises(ValueError, match="fp16 and bf16"):
        native.newton_schulz_group(xs[:2], xs[:2], shapes[:2], [native.NS_GRAM, native.NS_KELLER], ws, [None, None])


@pytest.mark.parametrize("blocks, rows, cols", [(4000, 66, 72), (1500, 72, 66), (700, 130, 257)])
def test_a_plan_of_many_tiles_equals_its_products_alone(blocks: int, rows: int, cols: int) -> None:
    """Hundreds of tiles per SM pair, each shorter than the way of its index to the pair's consumers: an
    entry of the tile ring that is written before it has been read everywhere shows as a wrong tile."""
    gen = torch.Generator(device=DEV).manual_seed(rows)
    x = torch.zeros(blocks, rows, _padded(cols), dtype=torch.float16, device=DEV)
    values = torch.randn(blocks, rows, cols, device=DEV, generator=gen)
    x[..., :cols] = values / values.norm(dim=(1, 2), keepdim=True)
    run = native.newton_schulz_tall if rows > cols else native.newton_schulz
    need = native.newton_schulz_tall_workspace_bytes if rows > cols else native.newton_schulz_workspace_bytes
    ws = torch.empty(need(blocks, rows, cols, native.NS_GRAM), dtype=torch.uint8, device=DEV)
    want, got = (torch.empty_like(x).view(torch.bfloat16) for _ in range(2))
    run(x.clone(), want, rows, cols, native.NS_GRAM + native.NS_STEPWISE, ws)
    for _ in range(3):
        run(x.clone(), got, rows, cols, native.NS_GRAM, ws)
        assert torch.equal(got[..., :cols], want[..., :cols])
    assert native.device_status() == 0


@pytest.mark.parametrize("blocks, rows, cols", [(1, 256, 520), (1, 500, 300), (2, 1000, 1100)])
def test_a_chain_of_one_matrix_reads_what_was_just_stored(blocks: int, rows: int, cols: int) -> None:
    """One or two matrices, so that every product starts the moment the one before it is stored: each lane of
    an epilogue warp must see the second term that other SMs wrote, iteration after iteration."""
    gen = torch.Generator(device=DEV).manual_seed(cols)
    x = torch.zeros(blocks, rows, _padded(cols), dtype=torch.float16, device=DEV)
    values = torch.randn(blocks, rows, cols, device=DEV, generator=gen)
    x[..., :cols] = values / values.norm(dim=(1, 2), keepdim=True)
    run = native.newton_schulz_tall if rows > cols else native.newton_schulz
    need = native.newton_schulz_tall_workspace_bytes if rows > cols else native.newton_schulz_workspace_bytes
    ws = torch.empty(need(blocks, rows, cols, native.NS_GRAM), dtype=torch.uint8, device=DEV)
    want = torch.empty_like(x).view(torch.bfloat16)
    run(x.clone(), want, rows, cols, native.NS_GRAM + native.NS_STEPWISE, ws)
    outs = []
    for i in range(64):
        ws.fill_(i)   # what the last iteration left in the scratch must not pass for this one's
        out = torch.empty_like(want)
        run(x.clone(), out, rows, cols, native.NS_GRAM, ws)
        outs.append(out)
    assert all(torch.equal(out[..., :cols], want[..., :cols]) for out in outs)
    assert native.device_status() == 0


@pytest.mark.parametrize("rows, cols", [(130, 257), (257, 130), (96, 96)])
def test_a_direct_call_can_leave_room_for_other_streams(rows: int, cols: int) -> None:
    """``stepwise``: one launch per product, the same result."""
    from dionw_b200.newton_schulz import NewtonSchulz, newton_schulz_fn

    gen = torch.Generator(device=DEV).manual_seed(rows)
    x = torch.randn(3, rows, cols, device=DEV, generator=gen)
    for kind in (NewtonSchulz.GRAM, NewtonSchulz.KELLER):
        call = newton_schulz_fn(kind)
        counts, outs = [], []
        for extra in ({}, {"stepwise": True}):
            before = native.launch_count()
            outs.append(call(x, 1e-8, **extra))
            counts.append(native.launch_count() - before)
        products = 18 if kind is NewtonSchulz.GRAM and rows != cols else 15
        assert counts[1] - counts[0] == products - 1
        assert torch.equal(*outs)


@pytest.mark.parametrize("rows, cols", [(9, 8), (8, 9)])
def test_more_blocks_than_a_grid_dimension_holds(rows: int, cols: int) -> None:
    """Either orientation takes any number of blocks; each comes out as it does in a small batch."""
    gen = torch.Generator(device=DEV).manual_seed(rows)
    blocks = 65536 + 9
    x = torch.zeros(blocks, rows, _padded(cols), dtype=torch.float16, device=DEV)
    x[..., :cols] = torch.randn(blocks, rows, cols, device=DEV, generator=gen) / 9.0
    run = native.newton_schulz_tall if rows > cols else native.newton_schulz
    need = native.newton_schulz_tall_workspace_bytes if rows > cols else native.newton_schulz_workspace_bytes
    ws = torch.empty(need(blocks, rows, cols, native.NS_GRAM), dtype=torch.uint8, device=DEV)
    out = torch.empty_like(x).view(torch.bfloat16)
    few = [x[:50].clone(), x[-50:].clone()]
    run(x, out, rows, cols, native.NS_GRAM, ws)
    for part, got in zip(few, (out[:50], out[-50:])):
        want = torch.empty_like(part).view(torch.bfloat16)
        run(part, want, rows, cols, native.NS_GRAM, ws)
        assert torch.equal(got[..., :cols], want[..., :cols])
    assert native.device_status() == 0


@pytest.mark.parametrize("update", ["DION3_UPDATE", "MUON_UPDATE"])
def test_a_step_in_groups_equals_a_step_run_by_run(update: str, monkeypatch: pytest.MonkeyPatch) -> None:
    import dionw_b200 as dionw

    shapes = [(1024, 1100), (1024, 1100), (96, 40), (40, 96), (64, 64), (1200, 1030), (8, 300), (33, 17), (20, 20)]
    results = []
    for group_max in (native.NS_GROUP_MAX, 1):
        monkeypatch.setattr(native, "NS_GROUP_MAX", group_max)
        gen = torch.Generator().manual_seed(11)
        model = torch.nn.ParameterList([torch.nn.Parameter((torch.randn(s, generator=gen) * 0.02).to(DEV)) for s in shapes])
        extra = {"fraction": 1.0} if update == "MUON_UPDATE" else {}
        optimizer = dionw.Dion(dionw.param_groups(model, **extra)[0], lr=1e-2, weight_decay=0.1,
                               matrix_update=getattr(dionw, update))
        for _ in range(3):
            for p in model:
                p.grad = (torch.randn(p.shape, generator=gen) * 1e-3).to(DEV)
            optimizer.step()
        results.append([t.clone() for p in model for t in (p.detach(), optimizer.state[p]["momentum"],
                                                           optimizer.state[p]["variance"])])
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("m", [100, 128, 129, 384, 385, 640, 641])
def test_symmetric_products_whose_last_narrow_tile_is_left_out(m: int) -> None:
    """Up to 128 columns into its last tile row a product of 128-wide tiles has no tile for the rest of it;
    one matrix and 300 of them, which take 128- and 256-wide tiles."""
    gen = torch.Generator().manual_seed(m)
    for blocks in (1, 300 if m <= 129 else 40):
        a = _operand(gen, blocks, m, 72, torch.float16)
        out = torch.full((blocks, m, _padded(m)), SENTINEL, dtype=torch.float16, device=DEV)
        native.symmetric_product(a[..., :72], out[..., :m])
        a64 = a[..., :72].double()
        _close(out[..., :m], a64 @ a64.mT, a64.abs() @ a64.mT.abs(), torch.float16)
        assert torch.equal(out[..., :m], out[..., :m].mT) and bool((out[..., m:] == SENTINEL).all())


@pytest.mark.parametrize("rows, cols, launches", [(64, 256, 18), (300, 64, 18), (64, 64, 15), (65, 256, 1), (65, 65, 1)])
def test_small_blocks_go_product_by_product(rows: int, cols: int, launches: int) -> None:
    """A plan's start costs more than it saves on them; in a group they are part of the plan all the same."""
    x = torch.zeros(2, rows, _padded(cols), dtype=torch.float16, device=DEV)
    x[..., :cols] = torch.randn(2, rows, cols, device=DEV, generator=torch.Generator(device=DEV).manual_seed(1)) / 64
    run = native.newton_schulz_tall if rows > cols else native.newton_schulz
    need = native.newton_schulz_tall_workspace_bytes if rows > cols else native.newton_schulz_workspace_bytes
    ws = torch.empty(need(2, rows, cols, native.NS_GRAM), dtype=torch.uint8, device=DEV)
    out = torch.empty_like(x).view(torch.bfloat16)
    before = native.launch_count()
    run(x.clone(), out, rows, cols, native.NS_GRAM, ws)
    assert native.launch_count() - before == launches
    shapes, kinds = [(2, rows, cols)] * 2, [native.NS_GRAM] * 2
    ws = torch.empty(native.newton_schulz_group_workspace_bytes(shapes, kinds), dtype=torch.uint8, device=DEV)
    xs = [x.clone(), x.clone()]
    before = native.launch_count()
    native.newton_schulz_group(xs, [v.view(torch.bfloat16) for v in xs], shapes, kinds, ws, [None, None])
    assert native.launch_count() - before == 1
    assert all(torch.equal(v.view(torch.bfloat16)[..., :cols], out[..., :cols]) for v in xs)
