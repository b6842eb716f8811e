"""The transient memory of a step: what lies where in a run's scratch, alone and in a group of runs."""

from __future__ import annotations

import pytest
import torch
from torch import nn

import dionw_b200 as dionw
from dionw_b200 import _matrix_step, _native, _workspace

# fused projection, projection, up and down of four 768-wide layers; a row-selecting pair beside them
SHAPES = [(768, 2304), (768, 768), (768, 3072), (3072, 768)] * 4 + [(1024, 2048)] * 2


def _described(monkeypatch: pytest.MonkeyPatch, update: str) -> list[tuple[_matrix_step.RunContext, _workspace.Plan]]:
    monkeypatch.setattr("dionw_b200.optimizer._require_param", lambda param: None)   # plans need no GPU
    model = nn.ParameterList([nn.Parameter(torch.zeros(shape)) for shape in SHAPES])
    extra = {"fraction": 1.0} if update == "MUON_UPDATE" else {}
    optimizer = dionw.Dion(dionw.param_groups(model, **extra)[0], lr=1e-3, matrix_update=getattr(dionw, update))
    for p in model:
        p.grad = torch.zeros_like(p)
    return [_matrix_step._describe_run(bucket, run, optimizer.param_groups[bucket.group_index])
            for bucket in optimizer._ensure_buckets() for run in optimizer._runs_of(bucket)]


def _bytes(plan: _workspace.Plan, names: list[str]) -> int:
    return sum(_workspace._round(torch.Size(plan[n][0]).numel() * plan[n][1].itemsize) for n in names)


@pytest.mark.parametrize("update", ["DION3_UPDATE", "MUON_UPDATE"])
def test_the_fp32_copies_of_a_group_lie_over_the_iterations_scratch(monkeypatch: pytest.MonkeyPatch, update: str) -> None:
    described = _described(monkeypatch, update)
    assert 1 < len(described) <= _native.NS_GROUP_MAX
    shapes = [(ctx.count, ctx.bucket.selected_rows, ctx.bucket.cols) for ctx, _ in described]
    kinds = [ctx.bucket.orthogonalize.code for ctx, _ in described]
    plan = _matrix_step._group_plan([own for _, own in described], shapes, kinds)
    offsets, total = _workspace.layout(plan)
    assert set(offsets) == {"ns"} | {f"{i}.{name}" for i, (_, own) in enumerate(described) for name in own}
    kept = sum(_bytes(own, [n for n in own if n != "u"]) for _, own in described)
    copies = [_bytes(own, ["u"]) for _, own in described if "u" in own]
    scratch = _native.newton_schulz_group_workspace_bytes(shapes, kinds)
    assert len(copies) >= 3
    assert total <= kept + _workspace._round(max(scratch, *copies))
    # nothing but copies and scratch shares bytes
    spans = sorted((start, start + size) for name, (start, size) in offsets.items() if not name.endswith(".u"))
    assert all(end <= start for (_, end), (start, _) in zip(spans, spans[1:]))
    start, size = offsets["ns"]
    assert all(offsets[n][0] == start and offsets[n][1] <= size for n in offsets if n.endswith(".u"))


def test_an_entry_over_a_shorter_one_is_refused() -> None:
    with pytest.raises(ValueError, match="has 8"):
        _workspace.layout({"a": ((2,), torch.float32), "b": ((3,), torch.float32, "a")})
