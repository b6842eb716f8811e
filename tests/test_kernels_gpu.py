"""Each CUDA entry point, called through the C ABI, against the CPU oracle."""

from __future__ import annotations

import math

import pytest
import torch

from conftest import PUBLISHED_ROUNDING, load_golden, rel_l2, spectrum_matrix as _spectrum_matrix
from oracle import dion_oracle as oracle

pytestmark = pytest.mark.gpu

DEV = "cuda"


@pytest.fixture(scope="module")
def native():
    from dionw_b200 import _native

    _native.library()
    return _native


def _gen(seed: int = 0) -> torch.Generator:
    return torch.Generator().manual_seed(seed)


# ---------------------------------------------------------------------------
# momentum passes
# ---------------------------------------------------------------------------
@pytest.mark.parametrize("shapes,cols", [([37], 3000), ([64, 64, 128], 4096), ([5], 1001), ([3, 1, 9], 520)])
def test_accumulate_row_l1_run_is_bit_exact(native, shapes, cols) -> None:
    """M exact; scores exact in the documented lane order (reference test:
    tests/test_momentum_kernels.py:10-19 allows rtol 1e-5 on the scores)."""
    g = _gen()
    grads = [torch.randn(r, cols, generator=g) for r in shapes]
    total = sum(shapes)
    momentum = torch.randn(total, cols, generator=g)
    expect_m = momentum.clone()
    expect_scores = []
    start = 0
    for grad in grads:
        expect_scores.append(oracle.accumulate_row_l1(grad, expect_m[start:start + grad.shape[0]], cols))
        start += grad.shape[0]
    expect_scores = torch.cat(expect_scores)
    m_dev = momentum.to(DEV)
    scores = torch.empty(total, device=DEV)
    sumsq = torch.empty(total, device=DEV)
    native.accumulate_row_l1_run([x.to(DEV) for x in grads], shapes, m_dev, scores, sumsq, cols)
    assert torch.equal(m_dev.cpu(), expect_m)
    assert torch.equal(scores.cpu(), expect_scores)
    assert torch.equal(sumsq.cpu(), oracle.row_sumsq(expect_m))
    torch.testing.assert_close(scores.cpu(), expect_m.abs().sum(-1), rtol=1e-5, atol=1e-3)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_accumulate_row_l1_run_casts_low_precision_grads(native, dtype) -> None:
    g = _gen(1)
    grad = torch.randn(16, 2048, generator=g).to(dtype)
    momentum = torch.randn(16, 2048, generator=g)
    expect = momentum + grad.float()
    m_dev = momentum.to(DEV)
    scores, sumsq = torch.empty(16, device=DEV), torch.empty(16, device=DEV)
    native.accumulate_row_l1_run([grad.to(DEV)], [16], m_dev, scores, sumsq, 2048)
    assert torch.equal(m_dev.cpu(), expect)
    assert torch.equal(scores.cpu(), oracle.row_scores(expect))


@pytest.mark.parametrize("nesterov", [False, True])
def test_accumulate_copy_decay_run(native, nesterov) -> None:
    """tests/test_momentum_kernels.py:22-42 of the reference (5001 elements)."""
    g = _gen(2)
    grad, momentum = torch.randn(1, 5001, generator=g), torch.randn(1, 5001, generator=g)
    expect_m = momentum.clone()
    expect_u = oracle.accumulate_copy_decay(grad, expect_m, 0.95, nesterov)
    m_dev, u = momentum.to(DEV), torch.empty(1, 5001, device=DEV)
    sumsq = torch.empty(1, device=DEV)
    native.accumulate_copy_decay_run([grad.to(DEV)], [1], m_dev, u, sumsq, 5001, 0.95, nesterov)
    assert torch.equal(m_dev.cpu(), expect_m)
    assert torch.equal(u.cpu(), expect_u)
    torch.testing.assert_close(sumsq.cpu(), expect_u.square().sum(-1), rtol=1e-5, atol=0)


@pytest.mark.parametrize("blocks,rows,k", [(3, 128, 32), (2, 14336, 3584), (1, 1000, 1), (2, 4096, 4096), (4, 257, 65)])
def test_select_rows_matches_oracle(native, blocks, rows, k) -> None:
    g = _gen(3)
    scores = torch.rand(blocks, rows, generator=g) + 0.5
    sumsq = torch.rand(blocks, rows, generator=g)
    expect = oracle.select_rows(scores, k)
    index = torch.empty(blocks, k, dtype=torch.int32, device=DEV)
    rowmap = torch.empty(blocks, rows, dtype=torch.int32, device=DEV)
    frob = torch.empty(blocks, device=DEV)
    native.select_rows(scores.to(DEV), sumsq.to(DEV), k, index, rowmap, frob)
    assert torch.equal(index.cpu().long(), expect)
    expect_map = torch.full((blocks, rows), -1, dtype=torch.int32)
    expect_map.scatter_(1, expect, torch.arange(k, dtype=torch.int32).expand(blocks, k))
    assert torch.equal(rowmap.cpu(), expect_map)
    torch.testing.assert_close(frob.cpu(), torch.gather(sumsq, 1, expect).sum(-1).sqrt(), rtol=1e-5, atol=0)


def test_select_rows_breaks_ties_toward_lower_rows(native) -> None:
    scores = torch.ones(1, 300)
    scores[0, 17] = 2.0
    scores[0, 250] = 0.5
    expect = oracle.select_rows(scores, 10)
    index = torch.empty(1, 10, dtype=torch.int32, device=DEV)
    rowmap = torch.empty(1, 300, dtype=torch.int32, device=DEV)
    frob = torch.empty(1, device=DEV)
    native.select_rows(scores.to(DEV), torch.ones(1, 300, device=DEV), 10, index, rowmap, frob)
    assert torch.equal(index.cpu().long(), expect)
    assert expect[0].tolist() == [0, 1, 2, 3, 4, 5, 6, 7, 8, 17]


@pytest.mark.parametrize("rows, k, above", [(9000, 4000, 700), (9000, 701, 700), (40001, 20000, 3), (40001, 40001, 9), (1025, 600, 0)])
def test_select_rows_breaks_ties_across_the_ctas_of_a_block(native, rows, k, above) -> None:
    """Two values, the lower one at the threshold and in the rows of every CTA of the cluster; 40001 rows are
    more than the CTAs keep in registers."""
    g = _gen(rows + k)
    scores = torch.full((2, rows), 0.5)
    scores.scatter_(1, torch.rand(2, rows, generator=g).topk(above).indices, 2.0)
    sumsq = torch.rand(2, rows, generator=g)
    expect = oracle.select_rows(scores, k)
    index = torch.empty(2, k, dtype=torch.int32, device=DEV)
    rowmap = torch.empty(2, rows, dtype=torch.int32, device=DEV)
    frob = torch.empty(2, device=DEV)
    native.select_rows(scores.to(DEV), sumsq.to(DEV), k, index, rowmap, frob)
    assert torch.equal(index.cpu().long(), expect)
    expect_map = torch.full((2, rows), -1, dtype=torch.int32)
    expect_map.scatter_(1, expect, torch.arange(k, dtype=torch.int32).expand(2, k))
    assert torch.equal(rowmap.cpu(), expect_map)
    # at most 40 additions per thread, 10 in the block, 8 over the cluster: 58 * 2^-24 of the sum, half of that of
    # its root, and the root's own rounding
    torch.testing.assert_close(frob.double().cpu(), torch.gather(sumsq, 1, expect).double().sum(-1).sqrt(),
                               rtol=60 * 2.0**-25, atol=0)


def test_select_rows_of_more_rows_than_stay_in_registers(native) -> None:
    g = _gen(12)
    scores, sumsq = torch.rand(1, 50003, generator=g) + 0.5, torch.rand(1, 50003, generator=g)
    expect = oracle.select_rows(scores, 12501)
    index = torch.empty(1, 12501, dtype=torch.int32, device=DEV)
    rowmap = torch.empty(1, 50003, dtype=torch.int32, device=DEV)
    frob = torch.empty(1, device=DEV)
    native.select_rows(scores.to(DEV), sumsq.to(DEV), 12501, index, rowmap, frob)
    assert torch.equal(index.cpu().long(), expect)


def test_pack_rows_decays_and_normalises(native) -> None:
    g = _gen(4)
    blocks, rows, k, cols = 2, 64, 16, 520
    momentum = torch.randn(blocks, rows, cols, generator=g)
    index = oracle.select_rows(torch.rand(blocks, rows, generator=g), k)
    picked = torch.gather(momentum, 1, index.unsqueeze(-1).expand(-1, -1, cols))
    frob = torch.linalg.vector_norm(picked, dim=(-2, -1))
    expect_x = (picked / (frob.view(-1, 1, 1) + 1e-8)).half()
    expect_m = momentum.clone()
    expect_m.scatter_(1, index.unsqueeze(-1).expand(-1, -1, cols), picked * 0.95)
    m_dev = momentum.to(DEV)
    x = torch.full((blocks, k, 520), float("nan"), dtype=torch.float16, device=DEV)
    native.pack_rows(m_dev, index.int().to(DEV), frob.to(DEV), k, x, decay=0.95, decay_rows=True, eps=1e-8)
    assert torch.equal(m_dev.cpu(), expect_m)
    assert torch.equal(x.cpu(), expect_x)


def test_transpose_2byte(native) -> None:
    src = torch.randn(3, 70, 130, generator=_gen(5)).half().to(DEV)
    dst = torch.empty(3, 130, 72, dtype=torch.float16, device=DEV)
    native.transpose_2byte(src, dst)
    assert torch.equal(dst[:, :, :70].cpu(), src.mT.cpu())
    assert float(dst[:, :, 70:].abs().max()) == 0.0


# ---------------------------------------------------------------------------
# tensor-core products
# ---------------------------------------------------------------------------
def _padded(t: torch.Tensor, ld: int) -> torch.Tensor:
    out = torch.zeros(*t.shape[:-1], ld, dtype=t.dtype, device=t.device)
    out[..., : t.shape[-1]] = t
    return out[..., : t.shape[-1]]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("blocks,m,kdim", [(3, 64, 256), (2, 300, 520), (1, 1024, 4096), (2, 384, 64), (1, 136, 72)])
def test_symmetric_product_aat(native, dtype, blocks, m, kdim) -> None:
    """ns_line_1 (src/dionw/_symmetric_kernels.py:252-277): fp32 accumulate, one rounding."""
    a = (torch.randn(blocks, m, kdim, generator=_gen(6)) / math.sqrt(kdim)).to(dtype).to(DEV)
    ld = (m + 7) // 8 * 8
    out = torch.full((blocks, m, ld), float("nan"), dtype=dtype, device=DEV)[..., :m]
    native.symmetric_product(a, out)
    assert native.device_status() == 0
    expect = (a.float() @ a.float().mT).to(dtype)
    assert rel_l2(out.float(), expect.float()) < 2e-3
    assert torch.equal(out, out.mT), "the stored product must be exactly symmetric"
    torch.testing.assert_close(out.float(), expect.float(), rtol=2e-2, atol=2e-3)


@pytest.mark.parametrize("m", [128, 200, 640])
def test_symmetric_product_polynomial_and_identity(native, m) -> None:
    """ns_line_2 plus the fused ``+ a I`` (src/dionw/_gram.py:60-63)."""
    base = torch.randn(2, m, m, generator=_gen(7)) / math.sqrt(m)
    sym = (base @ base.mT).half().to(DEV)
    sym = torch.triu(sym) + torch.triu(sym, 1).mT
    out = torch.empty_like(sym)
    out2 = torch.empty_like(sym)
    native.symmetric_product(sym, out, cin=sym, alpha=0.7, beta=-1.3, out2=out2, diag=float(torch.tensor(3.3).half()))
    assert native.device_status() == 0
    expect = (0.7 * (sym.float() @ sym.float().mT) - 1.3 * sym.float()).half()
    assert rel_l2(out.float(), expect.float()) < 2e-3
    expect2 = out + float(torch.tensor(3.3).half()) * torch.eye(m, dtype=torch.float16, device=DEV)
    assert torch.equal(out2, expect2)
    assert torch.equal(out, out.mT)


@pytest.mark.parametrize("m", [256, 520])
def test_symmetric_product_of_two_commuting_matrices(native, m) -> None:
    """``a Q + Q Z`` for polynomials Q, Z of one symmetric matrix (src/dionw/_gram.py:64-68):
    the lower triangle equals the general product, the upper one is its mirror."""
    base = torch.randn(2, m, m, generator=_gen(15)) / math.sqrt(m)
    g = base @ base.mT
    q = (0.3 * g + 0.5 * g @ g).half().to(DEV)
    z = (1.1 * g - 0.2 * g @ g @ g).half().to(DEV)
    q = torch.tril(q) + torch.tril(q, -1).mT
    z = torch.tril(z) + torch.tril(z, -1).mT
    out = torch.empty_like(q)
    native.symmetric_product(q, out, b=z, cin=q, alpha=1.0, beta=0.7)
    assert native.device_status() == 0
    general = torch.empty_like(q)
    native.batched_gemm(q, z, general, b_is_nk=True, cin=q, beta=0.7)
    assert torch.equal(torch.tril(out), torch.tril(general))
    assert torch.equal(out, out.mT)
    expect = (q.float() @ z.float() + 0.7 * q.float()).half()
    assert rel_l2(out.float(), expect.float()) < 2e-3


@pytest.mark.parametrize("b_is_nk", [True, False])
@pytest.mark.parametrize("blocks,m,n,kdim", [(2, 64, 256, 64), (1, 300, 520, 200), (2, 256, 1024, 256), (1, 128, 4096, 1024)])
def test_batched_gemm(native, b_is_nk, blocks, m, n, kdim) -> None:
    """torch.bmm / torch.baddbmm as used at src/dionw/_gram.py:58-69."""
    g = _gen(8)
    a = (torch.randn(blocks, m, kdim, generator=g) / math.sqrt(kdim)).half().to(DEV)
    b_kn = torch.randn(blocks, kdim, n, generator=g).half().to(DEV)
    cin = torch.randn(blocks, m, n, generator=g).half().to(DEV)
    b = b_kn.mT.contiguous() if b_is_nk else b_kn
    out = torch.empty(blocks, m, n, dtype=torch.float16, device=DEV)
    native.batched_gemm(a, b, out, b_is_nk=b_is_nk, cin=cin, beta=0.4)
    assert native.device_status() == 0
    expect = (a.float() @ b_kn.float() + 0.4 * cin.float()).half()
    assert rel_l2(out.float(), expect.float()) < 2e-3
    out_bf16 = torch.empty(blocks, m, n, dtype=torch.bfloat16, device=DEV)
    native.batched_gemm(a, b, out_bf16, b_is_nk=b_is_nk)
    assert rel_l2(out_bf16.float(), (a.float() @ b_kn.float())) < 5e-3


# ---------------------------------------------------------------------------
# Newton-Schulz
# ---------------------------------------------------------------------------
def _run_ns(native, x32: torch.Tensor, kind: int) -> torch.Tensor:
    """Normalise like the reference, run the device iteration on the wide orientation."""
    blocks, rows, cols = x32.shape
    tall = rows > cols
    wide = x32.mT.contiguous() if tall else x32
    m, n = wide.shape[1:]
    ld = (n + 7) // 8 * 8
    dtype = torch.float16 if kind in (0, 3) else torch.bfloat16
    if kind in (0, 3):
        xn = (wide / (torch.linalg.vector_norm(wide, dim=(-2, -1), keepdim=True) + 1e-8)).to(dtype)
    else:
        safety = 1.02 if kind == 1 else 1.0
        xb = wide.to(dtype)
        xn = xb / (xb.norm(dim=(-2, -1), keepdim=True) * safety + 1e-8)
    x = torch.zeros(blocks, m, ld, dtype=dtype, device=DEV)
    x[..., :n] = xn.to(DEV)
    ws = torch.empty(native.newton_schulz_workspace_bytes(blocks, m, n, kind), dtype=torch.uint8, device=DEV)
    out = torch.empty(blocks, m, ld, dtype=torch.bfloat16, device=DEV)
    native.newton_schulz(x, out, m, n, kind, ws)
    assert native.device_status() == 0
    result = out[..., :n].cpu()
    return result.mT if tall else result


@pytest.mark.parametrize("tag", ["wide", "tall", "square", "odd"])
def test_gram_newton_schulz_matches_reference_fixture(native, tag) -> None:
    """bf16 Newton-Schulz parity bound: rel-L2 <= 2e-3 is asked of weights; the
    iteration itself differs from the CPU run of the reference only by fp16
    accumulation order, checked here at 1e-2 on these tiny blocks and against
    the exact polar factor as the reference's own test does (< 0.2)."""
    gold = load_golden("newton_schulz")
    x = gold[f"{tag}.x"]
    ours = _run_ns(native, x, 0)
    assert ours.dtype == torch.bfloat16 and ours.shape == x.shape
    assert rel_l2(ours.float(), gold[f"{tag}.gram"].float()) < 1e-2
    assert rel_l2(ours.float(), oracle.exact_polar(x)) < 0.2


@pytest.mark.parametrize("blocks,m,n", [(2, 256, 4096), (1, 1024, 4096), (2, 512, 512), (1, 768, 2304)])
def test_gram_newton_schulz_matches_oracle(native, blocks, m, n) -> None:
    x = torch.randn(blocks, m, n, generator=_gen(9))
    ours = _run_ns(native, x, 0).float()
    torch.set_num_threads(8)
    expect = oracle.gram_newton_schulz(x).float()
    assert rel_l2(ours, expect) < 5e-3
    target = oracle.polynomial_fp64(x, eps=1e-8)
    assert rel_l2(ours, target) < 1.3 * rel_l2(expect, target) + 3e-3
    gram = ours.double() @ ours.double().mT
    eye = torch.eye(m, dtype=torch.float64)
    ref_gram = expect.double() @ expect.double().mT
    assert float((gram - eye).norm()) < 1.2 * float((ref_gram - eye).norm()) + 0.05


@pytest.mark.parametrize("blocks,m,n", [(2, 512, 2048), (1, 1024, 1280)])
def test_mirrored_gram_products_stay_within_the_rounding_of_the_full_ones(native, blocks, m, n) -> None:
    """GRAM mirrors ``aQ + QZ``, ``aG + GZ`` and ``aRZ + Z RZ`` (symmetric in exact arithmetic);
    GRAM_FULL computes them in full like the reference.  Both must sit at the same distance from
    the rounding-free polynomial and from an orthogonal matrix."""
    x = torch.randn(blocks, m, n, generator=_gen(16))
    mirrored = _run_ns(native, x, 0).float()
    full = _run_ns(native, x, 3).float()
    assert rel_l2(mirrored, full) < 1e-2  # nearly square operands amplify fp16 rounding either way
    target = oracle.polynomial_fp64(x, eps=1e-8)
    assert rel_l2(mirrored, target) < 1.3 * rel_l2(full, target) + 3e-3
    eye = torch.eye(m, dtype=torch.float64)
    err_m = float((mirrored.double() @ mirrored.double().mT - eye).norm())
    err_f = float((full.double() @ full.double().mT - eye).norm())
    assert err_m < 1.2 * err_f + 0.05


def _rounding_error(native, x: torch.Tensor, kind: int) -> float:
    if kind == 0:
        target = oracle.polynomial_fp64(x, oracle.GRAM_COEFFS, 1.0, eps=1e-7)
    else:
        target = oracle.polynomial_fp64(x, oracle.POLAR_EXPRESS_COEFFS, 1.02, eps=1e-7)
    ours = _run_ns(native, x, kind).double()
    return float((ours - target).norm() / target.norm())


@pytest.mark.parametrize("name", sorted(PUBLISHED_ROUNDING))
def test_gram_rounding_error_on_prescribed_spectra(native, name) -> None:
    x = _spectrum_matrix(name)
    ours = _rounding_error(native, x, 0)
    cpu = oracle.gram_newton_schulz(x, eps=1e-7).double()
    target = oracle.polynomial_fp64(x, oracle.GRAM_COEFFS, 1.0, eps=1e-7)
    cpu_error = float((cpu - target).norm() / target.norm())
    assert ours < PUBLISHED_ROUNDING[name] + 0.015, (ours, cpu_error)
    assert ours < 1.3 * cpu_error + 3e-3, (ours, cpu_error)
    if name != "gaussian":
        # the restart keeps the error of ill-conditioned inputs small, below bf16 Polar Express
        assert ours < 0.08
        if name != "geometric2":
            assert ours < _rounding_error(native, x, 1)


@pytest.mark.parametrize("name", ["geometric4", "geometric6", "lowrank3", "lowrank4"])
def test_fp32_input_beats_bf16_input_on_ill_conditioned_spectra(native, name) -> None:
    """The step hands the iteration fp32 momentum rows; rounding them to bf16 first (as
    microsoft/dion does) at least nearly doubles the error where singular values spread."""
    x = _spectrum_matrix(name)
    target = oracle.polynomial_fp64(x, oracle.GRAM_COEFFS, 1.0, eps=1e-7)
    from_fp32 = _rounding_error(native, x, 0)
    from_bf16 = float((_run_ns(native, x.bfloat16().float(), 0).double() - target).norm() / target.norm())
    assert from_bf16 > 1.8 * from_fp32, (from_bf16, from_fp32)


def _unit_bf16_batch(batch: int, m: int, n: int, seed: int) -> torch.Tensor:
    """The microbenchmark's input: N(0,1) entries, each matrix scaled to unit Frobenius norm, bf16."""
    x = torch.randn(batch, m, n, generator=_gen(seed))
    return (x / torch.linalg.matrix_norm(x, keepdim=True)).bfloat16()


@pytest.mark.parametrize("m,n", [(1024, 1024), (1024, 4096)])
def test_microbenchmark_batches_match_oracle_through_the_public_entry(native, m, n) -> None:
    """Batches of 16 bf16 matrices of unit Frobenius norm through ``gram_polar_express(x, 1e-8)``:
    the polar factors and the orthogonality error ``||Y Y^T - I||_F`` of two of the sixteen are
    compared with the CPU oracle, and every matrix of the batch must reach the same error level."""
    from dionw_b200.newton_schulz import gram_polar_express

    x = _unit_bf16_batch(16, m, n, seed=m + n)
    ours = gram_polar_express(x.to(DEV), 1e-8)
    assert native.device_status() == 0
    assert ours.dtype == torch.bfloat16 and ours.shape == x.shape
    ours = ours.float().cpu()
    torch.set_num_threads(8)
    expect = oracle.gram_newton_schulz(x[:2].float()).float()
    assert rel_l2(ours[:2], expect) < 5e-3
    eye = torch.eye(m, dtype=torch.float64)
    ref_err = [float((expect[i].double() @ expect[i].double().T - eye).norm()) for i in range(2)]
    our_err = [float((ours[i].double() @ ours[i].double().T - eye).norm()) for i in range(16)]
    for i in range(2):
        assert abs(our_err[i] - ref_err[i]) < 0.05 * ref_err[i] + 0.05
    assert max(our_err) < 1.2 * max(ref_err) + 0.05


@pytest.mark.parametrize("m,n,small_m,small_n", [(4096, 14336, 1024, 3584), (7168, 8192, 896, 1024)])
def test_large_operands_reach_the_orthogonality_of_small_ones(native, m, n, small_m, small_n) -> None:
    """4096 x 14336 (microbenchmark) and 7168 x 8192 (the gate/up operand of the 70B-shaped slice): the
    oracle would take minutes, but the error per sqrt(rows) is a property of the five fixed polynomial
    steps and the aspect ratio, not of the size, so it must stay at the level a small operand of the same
    aspect ratio reaches on the oracle."""
    from dionw_b200.newton_schulz import gram_polar_express

    small = _unit_bf16_batch(1, small_m, small_n, seed=5)
    torch.set_num_threads(8)
    expect = oracle.gram_newton_schulz(small.float()).double()[0]
    level = float((expect @ expect.T - torch.eye(small_m, dtype=torch.float64)).norm()) / small_m**0.5
    gen = torch.Generator(device=DEV).manual_seed(11)
    big = torch.randn(2, m, n, device=DEV, generator=gen)
    big = (big / torch.linalg.matrix_norm(big, keepdim=True)).bfloat16()
    y = gram_polar_express(big, 1e-8).float()
    assert native.device_status() == 0
    eye = torch.eye(m, device=DEV)
    for i in range(2):
        err = float(torch.linalg.matrix_norm(y[i] @ y[i].T - eye)) / m**0.5
        assert err < 1.25 * level + 0.01, (err, level)


@pytest.mark.parametrize("kind,name", [(1, "polar_express_triton"), (2, "keller_triton")])
@pytest.mark.parametrize("tag", ["wide", "tall", "square"])
def test_bf16_iterations_match_reference_fixture(native, kind, name, tag) -> None:
    gold = load_golden("newton_schulz")
    ours = _run_ns(native, gold[f"{tag}.x"], kind)
    assert rel_l2(ours.float(), gold[f"{tag}.{name}"].float()) < 3e-2


# ---------------------------------------------------------------------------
# NorMuon + apply
# ---------------------------------------------------------------------------
@pytest.mark.parametrize("selected", [True, False])
def test_normuon_and_apply_match_oracle(native, selected) -> None:
    g = _gen(10)
    blocks, rows, cols = 2, 96, 520
    k = 24 if selected else rows
    o = torch.randn(blocks, k, cols, generator=g).bfloat16() * 0.05
    variance = torch.rand(blocks, rows, 1, generator=g) * 1e-3
    weights = [torch.randn(rows, cols, generator=g) * 0.02 for _ in range(blocks)]
    index = oracle.select_rows(torch.rand(blocks, rows, generator=g), k) if selected else None
    step = -oracle.step_size(rows, cols, k, 3e-4)
    # oracle (src/dionw/_row_normalization.py:41-60, src/dionw/_matrix_step.py:274-304)
    v_sel = torch.gather(variance, 1, index.unsqueeze(-1)) if selected else variance
    update, v_new = oracle.normalize_rows(o, v_sel, 0.95, torch.tensor(step, dtype=torch.float32))
    expect_var = variance.clone()
    if selected:
        expect_var.scatter_(1, index.unsqueeze(-1), v_new)
    else:
        expect_var.copy_(v_new)
    factor = 1.0 - 3e-4 * 0.05
    expect_w = []
    for b, w in enumerate(weights):
        w = w * factor
        if selected:
            w.scatter_add_(0, index[b].unsqueeze(-1).expand(-1, cols), update[b])
        else:
            w.add_(update[b])
        expect_w.append(w)
    # device
    o_dev = o.to(DEV)
    s = torch.empty(blocks * k, device=DEV)
    native.row_sumsq_bf16(o_dev, cols, s)
    torch.testing.assert_close(s.cpu(), o.float().square().sum(-1).view(-1), rtol=1e-5, atol=0)
    var_dev = variance.view(blocks, rows).to(DEV)
    idx_dev = index.int().to(DEV) if selected else None
    rowmap = None
    if selected:
        rowmap = torch.full((blocks, rows), -1, dtype=torch.int32)
        rowmap.scatter_(1, index, torch.arange(k, dtype=torch.int32).expand(blocks, k))
        rowmap = rowmap.to(DEV)
    denom, scale = torch.empty(blocks * k, device=DEV), torch.empty(blocks, device=DEV)
    native.normuon_rows(s, var_dev, idx_dev, blocks=blocks, rows=rows, k=k, cols=cols, weight=1 - 0.95, eps=1e-8,
                        step=step, normalize=True, denom=denom, scale=scale)
    w_dev = [w.to(DEV) for w in weights]
    native.apply_run(w_dev, [rows] * blocks, o_dev, rowmap, denom, scale, rows=rows, k=k, cols=cols,
                     decay_factor=factor, has_decay=True)
    assert rel_l2(var_dev.cpu().view_as(expect_var), expect_var) < 1e-5
    for got, want in zip(w_dev, expect_w):
        assert rel_l2(got.cpu(), want) < 1e-6
    # rows that were not selected are decayed only, exactly
    if selected:
        mask = torch.ones(rows, dtype=torch.bool)
        mask[index[0]] = False
        assert torch.equal(w_dev[0].cpu()[mask], (weights[0] * torch.tensor(factor, dtype=torch.float32))[mask])


# ---------------------------------------------------------------------------
# AdamW and EMA
# ---------------------------------------------------------------------------
def test_adamw_multi_matches_torch_fused(native) -> None:
    """tests/test_optimizer.py:169-198 of the reference pins the AdamW route to
    torch.optim.AdamW(fused=True) exactly."""
    g = _gen(11)
    shapes = [(4096,), (1000, 33), (7,), (128256 // 8, 64)]
    params = [(torch.randn(s, generator=g) * 0.02).to(DEV) for s in shapes]
    ours = [p.clone() for p in params]
    theirs = [torch.nn.Parameter(p.clone()) for p in params]
    opt = torch.optim.AdamW(theirs, lr=3e-4, betas=(0.9, 0.95), weight_decay=0.05, eps=1e-8, fused=True)
    m = [torch.zeros_like(p) for p in ours]
    v = [torch.zeros_like(p) for p in ours]
    steps = [torch.zeros((), device=DEV) for _ in ours]
    for _ in range(3):
        grads = [(torch.randn(s, generator=g) * 1e-3).to(DEV) for s in shapes]
        for t, gr in zip(theirs, grads):
            t.grad = gr.clone()
        opt.step()
        native.adamw_multi(ours, grads, m, v, steps, lr=3e-4, beta1=0.9, beta2=0.95, weight_decay=0.05, eps=1e-8)
    for a, b in zip(ours, theirs):
        assert rel_l2(a, b.detach()) <= 1e-6
        torch.testing.assert_close(a, b.detach(), rtol=0, atol=0)
    assert all(float(s) == 3.0 for s in steps)


def test_adamw_multi_matches_fixture(native) -> None:
    gold = load_golden("adamw")
    p = gold["p0"].clone().to(DEV)
    m, v, step = torch.zeros_like(p), torch.zeros_like(p), torch.zeros((), device=DEV)
    for s in range(4):
        native.adamw_multi([p], [gold[f"g{s}"].to(DEV)], [m], [v], [step], lr=3e-4, beta1=0.9, beta2=0.95,
                           weight_decay=0.05, eps=1e-8)
        assert rel_l2(p, gold[f"p{s + 1}"]) <= 1e-5
        assert rel_l2(m, gold[f"m{s + 1}"]) <= 1e-5
        assert rel_l2(v, gold[f"v{s + 1}"]) <= 1e-5


def test_ema_multi_matches_lerp(native) -> None:
    g = _gen(12)
    sources = [torch.randn(n, generator=g).to(DEV) for n in (5, 4096 * 3, 100001)]
    shadows = [torch.zeros_like(s) for s in sources]
    native.ema_multi(shadows, sources, weight=0.0, first=True)
    for s, p in zip(shadows, sources):
        assert torch.equal(s, p)
    moved = [p + 0.1 for p in sources]
    expect = [s.clone().lerp_(p, 1.0 - 0.9999) for s, p in zip(shadows, moved)]
    native.ema_multi(shadows, moved, weight=1.0 - 0.9999, first=False)
    for s, e in zip(shadows, expect):
        torch.testing.assert_close(s, e, rtol=0, atol=0)
    # a constant parameter keeps a bit-exact shadow (tests/test_ema.py:287-305)
    frozen = [s.clone() for s in shadows]
    native.ema_multi(shadows, frozen, weight=0.3, first=False)
    for s, f in zip(shadows, frozen):
        assert torch.equal(s, f)


def test_ema_multi_upcasts_bf16_sources(native) -> None:
    src = torch.randn(3000, generator=_gen(13)).bfloat16().to(DEV)
    shadow = torch.zeros(3000, device=DEV)
    native.ema_multi([shadow], [src], weight=0.0, first=True)
    assert torch.equal(shadow, src.float())


def test_cpu_ema_job_updates_pinned_shadows(native) -> None:
    g = _gen(14)
    params = [torch.randn(n, generator=g).to(DEV) for n in (1000, 70000)]
    offsets = [0, 1000]
    staging_dev = torch.empty(71000, device=DEV)
    native.ema_stage_pack(params, offsets, staging_dev)
    staging_host = torch.empty(71000, pin_memory=True)
    staging_host.copy_(staging_dev, non_blocking=True)
    event = torch.cuda.Event()
    event.record()
    shadows = [torch.full((n,), 1.0) for n in (1000, 70000)]
    staged = [staging_host[0:1000], staging_host[1000:71000]]
    expect = [s.clone().lerp_(p.cpu(), 0.25) for s, p in zip(shadows, params)]
    job = native.CpuEmaJob(shadows, staged, [False, False], 0.25, event, threads=3)
    job.wait_copy()
    job.wait_update()
    assert job.done()
    job.close()
    for s, e in zip(shadows, expect):
        torch.testing.assert_close(s, e, rtol=0, atol=1e-7)


# ---------------------------------------------------------------------------
# row statistics from the last product's epilogue, one launch per round, device scalars, bounded waits
# ---------------------------------------------------------------------------
@pytest.mark.parametrize("kind,blocks,m,n", [(0, 2, 256, 4096), (0, 1, 1024, 1280), (0, 3, 200, 520), (0, 2, 512, 512),
                                             (1, 2, 384, 1000), (2, 1, 640, 640)])
def test_last_product_also_writes_the_row_sums_of_squares(native, kind, blocks, m, n) -> None:
    """``rowsq`` handed to the iteration comes back as partial sums per 128 columns whose total is the
    row's sum of squares of the bf16 output (what ``row_sumsq_bf16`` computes in a pass of its own),
    for the Gram schedule, the standard iteration and odd shapes; the output itself is unchanged."""
    x32 = torch.randn(blocks, m, n, generator=_gen(21))
    ld = (n + 7) // 8 * 8
    dtype = torch.float16 if kind == 0 else torch.bfloat16
    xn = (x32 / (torch.linalg.vector_norm(x32, dim=(-2, -1), keepdim=True) + 1e-8)).to(dtype)
    outs = []
    parts = native.newton_schulz_rowsq_parts(n)
    assert parts == 2 * ((n + 255) // 256)
    rowsq = torch.full((blocks * m, parts), float("nan"), device=DEV)
    for with_rowsq in (False, True):
        x = torch.zeros(blocks, m, ld, dtype=dtype, device=DEV)
        x[..., :n] = xn.to(DEV)
        ws = torch.empty(native.newton_schulz_workspace_bytes(blocks, m, n, kind), dtype=torch.uint8, device=DEV)
        out = torch.zeros(blocks, m, ld, dtype=torch.bfloat16, device=DEV)
        native.newton_schulz(x, out, m, n, kind, ws, rowsq if with_rowsq else None)
        outs.append(out)
    assert native.device_status() == 0
    assert torch.equal(outs[0], outs[1])
    assert not torch.isnan(rowsq).any()
    separate = torch.empty(blocks * m, device=DEV)
    native.row_sumsq_bf16(outs[1], n, separate)
    torch.testing.assert_close(rowsq.sum(dim=1), separate, rtol=2e-6, atol=0)
    exact = outs[1][..., :n].double().square().sum(-1).view(-1)
    torch.testing.assert_close(rowsq.double().sum(dim=1), exact, rtol=2e-6, atol=0)
    # NorMuon from the parts and from the whole sums: the same divisors and scales
    variance = torch.rand(blocks, m, generator=_gen(22)).to(DEV) * 1e-3
    results = []
    for s, p in ((rowsq, parts), (separate, 1)):
        v = variance.clone()
        denom, scale = torch.empty(blocks * m, device=DEV), torch.empty(blocks, device=DEV)
        native.normuon_rows(s, v, None, blocks=blocks, rows=m, k=m, cols=n, weight=0.05, eps=1e-8, step=-0.01,
                            normalize=True, denom=denom, scale=scale, parts=p)
        results.append((v, denom, scale))
    for a, b in zip(*results):
        torch.testing.assert_close(a, b, rtol=2e-6, atol=0)


def test_one_launch_applies_the_results_of_several_runs(native) -> None:
    """``apply_round`` over tensors whose update rows lie in three different buffers (what the ranks
    of a sharded round send) equals ``apply_run`` once per buffer, bit for bit -- with the decay
    factor passed as an argument, read from device memory, and with CTAs of four warps."""
    g = _gen(30)
    rows, cols, k = 96, 520, 24
    ld = (cols + 7) // 8 * 8
    factor = 1.0 - 3e-4 * 0.05
    runs = []
    for blocks_per_tensor in ([1, 2], [3], [1, 1, 1]):
        count = sum(blocks_per_tensor)
        o = torch.zeros(count, k, ld, dtype=torch.bfloat16)
        o[..., :cols] = torch.randn(count, k, cols, generator=g).bfloat16() * 0.05
        index = oracle.select_rows(torch.rand(count, rows, generator=g), k)
        rowmap = torch.full((count, rows), -1, dtype=torch.int32)
        rowmap.scatter_(1, index, torch.arange(k, dtype=torch.int32).expand(count, k))
        runs.append({"weights": [torch.randn(b * rows, cols, generator=g) * 0.02 for b in blocks_per_tensor],
                     "blocks": blocks_per_tensor, "o": o.to(DEV), "rowmap": rowmap.to(DEV),
                     "denom": (torch.rand(count * k, generator=g) + 0.5).to(DEV),
                     "scale": (torch.rand(count, generator=g) * -0.01).to(DEV)})
    expect = []
    for run in runs:
        w = [t.to(DEV) for t in run["weights"]]
        native.apply_run(w, [b * rows for b in run["blocks"]], run["o"], run["rowmap"], run["denom"], run["scale"],
                         rows=rows, k=k, cols=cols, decay_factor=factor, has_decay=True)
        expect += w
    device_factor = torch.tensor([factor], dtype=torch.float32, device=DEV)
    for decay_device, warps in ((None, 0), (device_factor, 0), (device_factor, 4)):
        weights, per_tensor, o, rowmap, denom, scale = [], [], [], [], [], []
        for run in runs:
            block = 0
            for t, b in zip(run["weights"], run["blocks"]):
                weights.append(t.to(DEV))
                per_tensor.append(b * rows)
                o.append(run["o"][block].data_ptr())
                rowmap.append(run["rowmap"][block].data_ptr())
                denom.append(run["denom"][block * k:].data_ptr())
                scale.append(run["scale"][block:].data_ptr())
                block += b
        native.apply_round(weights, per_tensor, o, rowmap, denom, scale, ldo=ld, rows=rows, k=k, cols=cols,
                           decay_factor=123.0 if decay_device is not None else factor, has_decay=True,
                           decay_device=decay_device, cta_warps=warps)
        for got, want in zip(weights, expect):
            assert torch.equal(got, want)


def test_adamw_and_normuon_read_their_scalars_from_device_memory(native) -> None:
    """lr and weight decay of AdamW, and the step of NorMuon, taken from device memory give the bits
    of the same values passed as arguments; ``write_scalars`` is ordered on the stream."""
    g = _gen(31)
    table = torch.zeros(600, device=DEV)
    values = [float(v) for v in torch.rand(600, generator=g)]
    native.write_scalars(table, values)
    assert torch.equal(table.cpu(), torch.tensor(values, dtype=torch.float32))
    native.write_scalars(table, [3e-4, 0.05, -0.0123])
    n = 5000
    start = [torch.randn(n, generator=g) * 0.02 for _ in range(4)]
    outs = []
    for hyper in (None, table[:2]):
        p, grad, m, v = (t.to(DEV).clone() for t in start)
        v = v.abs()
        steps = torch.zeros((), device=DEV)
        for _ in range(2):
            native.adamw_multi([p], [grad], [m], [v], [steps], lr=3e-4 if hyper is None else 9.0, beta1=0.9,
                               beta2=0.95, weight_decay=0.05 if hyper is None else 9.0, eps=1e-8, hyper_device=hyper)
        outs.append((p, m, v))
    for a, b in zip(*outs):
        assert torch.equal(a, b)
    s = torch.rand(2 * 40, generator=g).to(DEV)
    scales = []
    for step_device in (None, table[2:3]):
        variance = torch.zeros(2, 40, device=DEV)
        denom, scale = torch.empty(80, device=DEV), torch.empty(2, device=DEV)
        native.normuon_rows(s, variance, None, blocks=2, rows=40, k=40, cols=64, weight=0.05, eps=1e-8,
                            step=-0.0123 if step_device is None else 5.0, normalize=True, denom=denom, scale=scale,
                            step_device=step_device)
        scales.append(scale)
    assert torch.equal(scales[0], scales[1])


def test_a_wait_that_runs_out_is_reported_and_the_device_stays_usable(native) -> None:
    """The tensor-core kernels bound every wait on a barrier.  The library's self-test kernel waits
    one millisecond on a barrier nothing arrives on, with the products' own wait routine: it must
    RETURN, leave the wait code in the device status word, ``check_device`` must raise once, and an
    ordinary product right after must be correct."""
    assert native.device_status() == 0
    gave_up = torch.zeros((), dtype=torch.int32, device=DEV)
    native.selftest_wait_timeout(1000, gave_up)
    torch.cuda.synchronize()
    assert int(gave_up) == 1
    with pytest.raises(native.DeviceWaitError, match="0x7001"):
        native.check_device()
    native.check_device()   # the word was cleared by the read
    a = (torch.randn(2, 300, 520, generator=_gen(5)) / 520**0.5).half().to(DEV)
    out = torch.empty(2, 300, 304, dtype=torch.float16, device=DEV)
    native.symmetric_product(a, out)
    torch.cuda.synchronize()
    expect = a.float() @ a.float().mT
    assert rel_l2(out[..., :300], expect) < 2e-3
    assert native.device_status() == 0


def test_tiles_drawn_from_a_counter_give_the_same_bits(native) -> None:
    """Multi-wave products with their tiles handed out by a device counter (the form used beside
    NCCL's kernels in the sharded step) against the fixed stride: symmetric and general schedules,
    several launches in a row on one stream (each launch must leave the counters at zero for the
    next) and launches of two streams in flight together (each stream has counters of its own)."""
    g = _gen(40)
    a = (torch.randn(5, 1536, 512, generator=g) / 512**0.5).half().to(DEV)        # 5 x 21 = 105 tiles of the triangle
    x = (torch.randn(3, 1024, 512, generator=g) / 512**0.5).half().to(DEV)
    w = torch.randn(3, 512, 2560, generator=g).half().to(DEV)                     # 3 x 4 x 10 = 120 tiles

    def products(stream=None):
        sym = torch.empty(5, 1536, 1536, dtype=torch.float16, device=DEV)
        gen = torch.empty(3, 1024, 2560, dtype=torch.float16, device=DEV)
        with torch.cuda.stream(stream or torch.cuda.current_stream()):
            for _ in range(3):
                native.symmetric_product(a, sym)
                native.batched_gemm(x, w, gen, b_is_nk=False)
        return sym, gen

    was = native.gemm_dynamic_tiles(False)
    try:
        expect = products()
        torch.cuda.synchronize()
        assert native.gemm_dynamic_tiles(True) is False
        got = products()
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        beside = products(side)
        again = products()
        torch.cuda.synchronize()
        assert native.device_status() == 0
        for result in (got, beside, again):
            for mine, want in zip(result, expect):
                assert torch.equal(mine, want)
        assert rel_l2(got[0], a.float() @ a.float().mT) < 2e-3
    finally:
        native.gemm_dynamic_tiles(was)


def test_products_decay_unselected_rows_while_they_wait(native) -> None:
    """A decay job carried by a long product: its epilogue warps multiply unselected rows of the job's
    weights by the decay factor while they wait; the update kernel given the same job skips those and
    does the rest.  The weights equal, bit for bit, the update kernel doing all of it -- whatever
    share of the rows the product got to (here it must get to some)."""
    g = _gen(50)
    rows, cols, k = 512, 1024, 128
    ld = cols
    factor = 1.0 - 3e-4 * 0.05
    blocks_per_tensor = [2, 1, 3]
    count = sum(blocks_per_tensor)
    o = (torch.randn(count, k, ld, generator=g) * 0.05).bfloat16().to(DEV)
    index = oracle.select_rows(torch.rand(count, rows, generator=g), k)
    rowmap = torch.full((count, rows), -1, dtype=torch.int32)
    rowmap.scatter_(1, index, torch.arange(k, dtype=torch.int32).expand(count, k))
    rowmap = rowmap.to(DEV)
    denom = (torch.rand(count * k, generator=g) + 0.5).to(DEV)
    scale = (torch.rand(count, generator=g) * -0.01).to(DEV)
    start = [torch.randn(b * rows, cols, generator=g) * 0.02 for b in blocks_per_tensor]
    per_tensor = [b * rows for b in blocks_per_tensor]

    def tables(weights):
        o_p, m_p, d_p, s_p, block = [], [], [], [], 0
        for b in blocks_per_tensor:
            o_p.append(o[block].data_ptr()); m_p.append(rowmap[block].data_ptr())
            d_p.append(denom[block * k:].data_ptr()); s_p.append(scale[block:].data_ptr())
            block += b
        return o_p, m_p, d_p, s_p

    expect = [t.to(DEV) for t in start]
    o_p, m_p, d_p, s_p = tables(expect)
    native.apply_round(expect, per_tensor, o_p, m_p, d_p, s_p, ldo=ld, rows=rows, k=k, cols=cols,
                       decay_factor=factor, has_decay=True)
    got = [t.to(DEV) for t in start]
    job = torch.zeros(native.decay_job_bytes(), dtype=torch.uint8, device=DEV)
    native.decay_job_begin(job, got, m_p, per_tensor, rows=rows, cols=cols, decay_factor=factor, rows_per_wait=2)
    a = (torch.randn(4, 1536, 4096, generator=g) / 64).half().to(DEV)     # K = 4096: a long main loop, 84 tiles
    out = torch.empty(4, 1536, 1536, dtype=torch.float16, device=DEV)
    plain = torch.empty_like(out)
    native.symmetric_product(a, plain)
    native.gemm_side_job(job)
    try:
        native.symmetric_product(a, out)
    finally:
        native.gemm_side_job(None)
    torch.cuda.synchronize()
    taken = int(job[20:24].view(torch.int32))
    assert taken > 0, "the product's epilogue warps took no row of the job"
    assert torch.equal(out, plain)
    half_done = [t.clone() for t in got]
    native.apply_round(got, per_tensor, o_p, m_p, d_p, s_p, ldo=ld, rows=rows, k=k, cols=cols,
                       decay_factor=factor, has_decay=True, decay_job=job)
    torch.cuda.synchronize()
    assert native.device_status() == 0
    for mine, want in zip(got, expect):
        assert torch.equal(mine, want)
    # what the product did: unselected rows below the cursor are decayed exactly once, nothing else is touched
    flat_map = rowmap.view(-1).cpu()
    before, after = torch.cat(start), torch.cat([t.cpu() for t in half_done])
    done = min(taken, before.shape[0])
    unselected = flat_map[:done] < 0
    assert torch.equal(after[:done][unselected], before[:done][unselected] * torch.tensor(factor, dtype=torch.float32))
    assert torch.equal(after[:done][~unselected], before[:done][~unselected])
    assert torch.equal(after[done:], before[done:])
