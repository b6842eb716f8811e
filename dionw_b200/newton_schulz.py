"""The orthogonalization of matrix updates (src/dionw/newton_schulz.py:33-68).

Every kind runs five quintic steps on a batch of matrices and returns bfloat16.
All of them run on this package's tcgen05 kernels: ``GRAM`` in float16 with the
Gram schedule of src/dionw/_gram.py:41-89, the Polar Express and Keller kinds in
bfloat16 with the schedule of src/dionw/_polar_express.py:74-104 (the ``_TRITON``
and plain names select the same device code here; the enum keeps both values
because they are part of the checkpoint's structural keys).
"""

from __future__ import annotations

import enum
from collections.abc import Callable
from dataclasses import dataclass

import torch
from torch import Tensor

from dionw_b200 import _native

# ([N, rows, cols] batch, epsilon added to the Frobenius norm) -> bf16 polar factors
Orthogonalize = Callable[[Tensor, float], Tensor]


class NewtonSchulz(enum.Enum):
    """Which iteration orthogonalizes matrix updates."""

    POLAR_EXPRESS = "polar_express"
    POLAR_EXPRESS_TRITON = "polar_express_triton"
    GRAM = "gram"
    KELLER = "keller"
    KELLER_TRITON = "keller_triton"


def padded(n: int) -> int:
    """Leading dimension used for 2-byte operands: a multiple of 8 elements (16 bytes)."""
    return (n + 7) // 8 * 8


@dataclass(frozen=True)
class NativeOrthogonalizer:
    """A built-in iteration.  ``Dion`` recognises it and feeds it from its fused
    pack kernel; called directly it orthogonalizes any ``[N, rows, cols]`` batch.

    A direct call is one launch that holds every SM until the iteration is done.  With
    ``stepwise=True`` it is one launch per product, between which kernels of other streams
    (collectives, a data loader's copies) get SMs; the result is the same bit for bit.
    """

    kind: NewtonSchulz
    code: int             # DIONW_NS_* of the C ABI
    dtype: torch.dtype    # element type of the iteration
    norm_scale: float     # factor on the Frobenius norm before normalising

    def __call__(self, matrix: Tensor, epsilon: float, *, stepwise: bool = False) -> Tensor:
        if matrix.ndim != 3:
            raise ValueError(f"expected a [N, rows, cols] batch, got shape {tuple(matrix.shape)}")
        if not matrix.is_cuda:
            raise ValueError("dionw_b200 orthogonalizes on CUDA devices only")
        blocks, rows, cols = matrix.shape
        src = matrix if matrix.dtype in (torch.float32, torch.float16, torch.bfloat16) else matrix.float()
        src = src.contiguous()
        x = torch.empty(blocks, rows, padded(cols), dtype=self.dtype, device=src.device)
        _native.normalize_pack(src, x, eps=epsilon, norm_scale=self.norm_scale)
        scratch = torch.empty(self.workspace_bytes(blocks, rows, cols), dtype=torch.uint8, device=src.device)
        out = run_iteration(self, x, rows, cols, scratch, stepwise=stepwise)
        return out[..., :cols]

    def workspace_bytes(self, blocks: int, rows: int, cols: int) -> int:
        if rows > cols:
            return _native.newton_schulz_tall_workspace_bytes(blocks, rows, cols, self.code)
        return _native.newton_schulz_workspace_bytes(blocks, rows, cols, self.code)


def run_iteration(fn: NativeOrthogonalizer, x: Tensor, rows: int, cols: int, scratch: Tensor,
                  rowsq: Tensor | None = None, stepwise: bool = False) -> Tensor:
    """Iterate in place on ``x`` ``[N, rows, ld]`` (normalised, in ``fn.dtype``); returns bf16 ``[N, rows, ld]``.

    ``scratch`` holds ``fn.workspace_bytes(...)`` bytes.  ``rowsq``: fp32
    ``[N * rows, newton_schulz_rowsq_parts(cols)]``, filled with partial row
    sums of the squared result by the last product's epilogue.  ``stepwise``: one
    launch per product, for a call that runs beside other streams' kernels.
    """
    out = x if x.dtype is torch.bfloat16 else x.view(torch.bfloat16)
    iterate = _native.newton_schulz_tall if rows > cols else _native.newton_schulz
    iterate(x, out, rows, cols, fn.code + (_native.NS_STEPWISE if stepwise else 0), scratch, rowsq)
    return out


_NATIVE = {
    NewtonSchulz.GRAM: NativeOrthogonalizer(NewtonSchulz.GRAM, _native.NS_GRAM, torch.float16, 1.0),
    NewtonSchulz.POLAR_EXPRESS: NativeOrthogonalizer(
        NewtonSchulz.POLAR_EXPRESS, _native.NS_POLAR_EXPRESS, torch.bfloat16, 1.02),
    NewtonSchulz.POLAR_EXPRESS_TRITON: NativeOrthogonalizer(
        NewtonSchulz.POLAR_EXPRESS_TRITON, _native.NS_POLAR_EXPRESS, torch.bfloat16, 1.02),
    NewtonSchulz.KELLER: NativeOrthogonalizer(NewtonSchulz.KELLER, _native.NS_KELLER, torch.bfloat16, 1.0),
    NewtonSchulz.KELLER_TRITON: NativeOrthogonalizer(
        NewtonSchulz.KELLER_TRITON, _native.NS_KELLER, torch.bfloat16, 1.0),
}


def newton_schulz_fn(kind: NewtonSchulz) -> Orthogonalize:
    """The orthogonalization for ``kind``.

    Raises:
        RuntimeError: For an unhandled kind.
    """
    try:
        return _NATIVE[kind]
    except KeyError:
        raise RuntimeError(f"Unhandled NewtonSchulz: {kind}") from None


def gram_polar_express(matrix: Tensor, epsilon: float) -> Tensor:
    """Gram Newton-Schulz of a batch, bf16 (src/dionw/_gram.py:72-89)."""
    return _NATIVE[NewtonSchulz.GRAM](matrix, epsilon)
