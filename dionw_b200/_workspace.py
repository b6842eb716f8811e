"""Per-device scratch arenas for the transient buffers of a run.

One byte tensor per (device, arena name), grown when a run needs more and
reused by every later run and step: runs execute one after another on one
stream, so they can share it, and the caching allocator is not asked for
gigabytes every step.  A plan is an ordered ``name -> (shape, dtype)`` mapping;
its entries are laid out in order, each starting on a 256-byte boundary, so two
processes that build the same plan agree on every offset.  An entry ``(shape,
dtype, other)`` lies over the start of the earlier entry ``other``, which is at
least as long: the two are not in use at the same time.
"""

from __future__ import annotations

import math

import torch
from torch import Tensor

_ALIGN = 256
_arenas: dict[tuple[torch.device, str], Tensor] = {}
# The views of recent plans, which a training loop carves again every step: making a dozen typed views
# costs 60 us of host time, looking them up 5.  Dropped whenever an arena changes; at most _CARVED_MAX.
_carved: dict[tuple[object, ...], dict[str, Tensor]] = {}
_CARVED_MAX = 64
# Bumped whenever an arena is allocated, regrown or dropped: a recorded CUDA graph holds arena
# addresses and is only valid while this number stands.
generation = 0

Plan = dict[str, tuple[tuple[int, ...], torch.dtype] | tuple[tuple[int, ...], torch.dtype, str]]


def _round(n: int) -> int:
    return (n + _ALIGN - 1) // _ALIGN * _ALIGN


def layout(plan: Plan) -> tuple[dict[str, tuple[int, int]], int]:
    """``name -> (byte offset, byte size)`` of every entry, and the total bytes."""
    offsets: dict[str, tuple[int, int]] = {}
    cursor = 0
    for name, (shape, dtype, *over) in plan.items():
        nbytes = math.prod(shape) * dtype.itemsize
        if over:
            start, room = offsets[over[0]]
            if nbytes > room:
                raise ValueError(f"{name} needs {nbytes} bytes, {over[0]} under it has {room}")
            offsets[name] = (start, nbytes)
            continue
        offsets[name] = (cursor, nbytes)
        cursor += _round(nbytes)
    return offsets, cursor


def views(buffer: Tensor, plan: Plan, base: int = 0) -> dict[str, Tensor]:
    """Typed views of ``buffer`` (a byte tensor) for every entry of ``plan``, laid out from ``base``."""
    offsets, _ = layout(plan)
    out: dict[str, Tensor] = {}
    for name, (shape, dtype, *_) in plan.items():
        start, nbytes = offsets[name]
        out[name] = buffer[base + start : base + start + nbytes].view(dtype).view(shape)
    return out


def arena(device: torch.device, nbytes: int, name: str = "run") -> Tensor:
    """The named byte arena of ``device``, at least ``nbytes`` long (contents unspecified)."""
    key = (device, name)
    buffer = _arenas.get(key)
    if buffer is None or buffer.numel() < nbytes:
        global generation
        generation += 1
        _carved.clear()
        _arenas.pop(key, None)
        buffer = torch.empty(max(nbytes, 1 << 20), dtype=torch.uint8, device=device)
        _arenas[key] = buffer
    return buffer


def carve(device: torch.device, plan: Plan, name: str = "run") -> dict[str, Tensor]:
    """One tensor per plan entry, all views of the device's arena ``name``."""
    key = (device, name, tuple(plan.items()))
    found = _carved.get(key)
    if found is None:
        _, total = layout(plan)
        found = views(arena(device, total, name), plan)   # may drop what was carved before
        if len(_carved) >= _CARVED_MAX:
            _carved.clear()
        _carved[key] = found
    return found


def release() -> None:
    """Drop every arena (tests, or before a memory-hungry phase)."""
    global generation
    generation += 1
    _carved.clear()
    _arenas.clear()
