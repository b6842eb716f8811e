"""The iteration of small blocks on chip, and symmetric matrices stored up to the diagonal, where they can go wrong.

Both keep the bits of the products run one by one, which the other tests hold to the oracle: the same
instructions on the same values in the same order, the same triangle mirrored.
"""

from __future__ import annotations

import pytest
import torch

from dionw_b200 import _native as native
from oracle import dion_oracle as oracle

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
STEPWISE = native.NS_STEPWISE


def _operand(blocks: int, rows: int, cols: int, dtype: torch.dtype = torch.float16) -> torch.Tensor:
    x = torch.zeros(blocks, rows, (cols + 7) // 8 * 8, dtype=dtype, device=DEV)
    values = torch.randn(blocks, rows, cols, device=DEV, generator=torch.Generator(device=DEV).manual_seed(rows + cols))
    x[..., :cols] = (values / values.norm(dim=(1, 2), keepdim=True)).to(dtype)
    return x


def _iterate(x: torch.Tensor, cols: int, kind: int, fill: int = 255) -> tuple[torch.Tensor, torch.Tensor]:
    """The result and its row sums, with every byte of the scratch `fill` (255: not a number) beforehand."""
    blocks, rows, _ = x.shape
    tall = rows > cols
    need = native.newton_schulz_tall_workspace_bytes if tall else native.newton_schulz_workspace_bytes
    ws = torch.full((need(blocks, rows, cols, kind & ~STEPWISE),), fill, dtype=torch.uint8, device=DEV)
    out = torch.full_like(x, 77.0).view(torch.bfloat16)
    sums = torch.full((blocks * rows, native.newton_schulz_rowsq_parts(cols)), 77.0, device=DEV)
    (native.newton_schulz_tall if tall else native.newton_schulz)(x.clone(), out, rows, cols, kind, ws, sums)
    return out[..., :cols], sums


# m at the edges of a 16-wide step, of 32-wide pieces, 64-wide panels and images, and of the second CTA's rows; n at
# the edges of 64-wide k-blocks and 256-wide tiles, with one to eight pairs to a matrix, tiles for some of them only,
# and more matrices than clusters that run at a time
@pytest.mark.parametrize("blocks, m, n", [
    (1, 65, 66), (2, 79, 257), (3, 80, 81), (1, 95, 1000), (2, 96, 512), (1, 97, 513), (2, 127, 128), (2, 128, 129),
    (1, 128, 1024), (3, 129, 130), (2, 130, 600), (1, 159, 300), (2, 160, 2049), (1, 161, 256), (2, 191, 700), (1, 192, 193),
    (3, 193, 1025), (1, 224, 225), (2, 225, 800), (1, 255, 256), (2, 255, 777), (1, 256, 257), (4, 256, 1024), (20, 200, 600),
    (40, 256, 300), (80, 66, 70), (200, 130, 140), (1, 66, 6144), (1, 66, 6145), (75, 70, 1024), (75, 70, 1025)])
@pytest.mark.parametrize("tall", [False, True])
def test_small_blocks_on_chip_have_the_bits_of_their_products(blocks: int, m: int, n: int, tall: bool) -> None:
    rows, cols = (n, m) if tall else (m, n)
    x = _operand(blocks, rows, cols)
    want, want_sums = _iterate(x, cols, native.NS_GRAM + STEPWISE)
    # Columns that make a matrix too wide to be the faster on chip: 6144, and 1024 where a wave of pairs is too small.
    wave = torch.cuda.get_device_properties(DEV).multi_processor_count // 2
    pairs = native.newton_schulz_on_chip_pairs(blocks, rows, cols, native.NS_GRAM)
    assert (pairs > 0) == (n <= (6144 if blocks <= wave else 1024))
    assert pairs <= -(-n // 256) and (pairs > 1 or blocks > 1 or n <= 256 or n > 6144)
    before = native.launch_count()
    got, sums = _iterate(x, cols, native.NS_GRAM)
    assert native.launch_count() - before == 1
    assert torch.equal(got, want) and torch.equal(sums, want_sums)
    for _ in range(3):   # what could differ is the order in which warps, copies and CTAs get through
        again, sums = _iterate(x, cols, native.NS_GRAM)
        assert torch.equal(again, want) and torch.equal(sums, want_sums)
    assert native.device_status() == 0


def test_what_is_not_iterated_on_chip() -> None:
    pairs = native.newton_schulz_on_chip_pairs
    assert pairs(1, 256, 4096, native.NS_GRAM) == pairs(1, 4096, 256, native.NS_GRAM) == 8
    for kind in (native.NS_GRAM + STEPWISE, native.NS_GRAM_FULL, native.NS_POLAR_EXPRESS, native.NS_KELLER):
        assert pairs(1, 256, 4096, kind) == 0
    for blocks, rows, cols in ((1, 257, 1024), (1, 64, 1024), (1, 256, 256), (20000, 96, 128), (0, 256, 1024)):
        assert pairs(blocks, rows, cols, native.NS_GRAM) == 0


def test_small_blocks_on_chip_in_two_streams() -> None:
    """Clusters of two launches side by side: nothing of an iteration lies outside its own buffers."""
    x = _operand(6, 200, 900)
    want, _ = _iterate(x, 900, native.NS_GRAM + STEPWISE)
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    outs = []
    for i in range(8):
        with torch.cuda.stream(streams[i % 2]):
            outs.append(_iterate(x, 900, native.NS_GRAM)[0])
    torch.cuda.synchronize()
    assert all(torch.equal(out, want) for out in outs)


# one to three 256-row blocks, full and with a remainder: what lies right of the diagonal blocks is never written, and
# the scratch is not-a-number, so that a result that read it would be too
@pytest.mark.parametrize("kind", [native.NS_GRAM, native.NS_KELLER])
@pytest.mark.parametrize("rows, cols", [(257, 700), (700, 257), (384, 384), (511, 700), (512, 800), (800, 513), (640, 1100), (1000, 769)])
def test_nothing_reads_past_the_diagonal_blocks(rows: int, cols: int, kind: int) -> None:
    x = _operand(2, rows, cols, torch.float16 if kind == native.NS_GRAM else torch.bfloat16)
    got, _ = _iterate(x, cols, kind)
    assert torch.equal(got, _iterate(x, cols, kind, fill=0)[0])
    assert torch.equal(got, _iterate(x, cols, kind + STEPWISE)[0])
    table = oracle.GRAM_COEFFS if kind == native.NS_GRAM else oracle.KELLER_COEFFS
    target = oracle.polynomial_fp64(x[..., :cols].float().cpu(), table, 1.0, eps=1e-8)
    def distance(result: torch.Tensor) -> float:
        return float((result.double().cpu() - target).norm() / target.norm())

    if kind == native.NS_GRAM and rows != cols:
        # GRAM_FULL stores and reads whole matrices: the bound that mirrored products are held to elsewhere.  (Sides at least
        # a quarter apart: the nearer to square, the more rounding is amplified, for mirrored and full products differently.)
        assert distance(got) < 1.3 * distance(_iterate(x, cols, native.NS_GRAM_FULL)[0]) + 3e-3
    else:
        # five steps without a restart, each rounded to 2^-11 (2^-8) of a matrix of norm near 1: some 2^-9 (2^-6) in all
        assert distance(got) < 2 * (2.0**-9 if kind == native.NS_GRAM else 2.0**-6)
