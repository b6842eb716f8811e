"""DIONW_GEMM_PDL=0 turns programmatic dependence off for every kernel of a step.  The switch is read once
per process, so a child process records a step into a CUDA graph and counts the graph's programmatic edges."""

from __future__ import annotations

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import torch
from cuda.bindings import runtime as cuda
import dionw_b200 as dionw
gen = torch.Generator().manual_seed(0)
shapes = [(1024, 1100), (96, 40), (64, 64), (33,)]
model = torch.nn.ParameterList([torch.nn.Parameter((torch.randn(s, generator=gen) * 0.02).cuda()) for s in shapes])
optimizer = dionw.Dion(dionw.param_groups(model)[0], lr=1e-2)
for p in model:
    p.grad = torch.full_like(p, 1e-3)
optimizer.step()
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph(keep_graph=True)
with torch.cuda.graph(graph):
    optimizer.step()
handle = cuda.cudaGraph_t(graph.raw_cuda_graph())
err, *_, count = cuda.cudaGraphGetEdges_v2(handle)
assert int(err) == 0, err
err, _, _, data, count = cuda.cudaGraphGetEdges_v2(handle, count)
assert int(err) == 0, err
print("EDGES", sum(edge.type == cuda.cudaGraphDependencyType.cudaGraphDependencyTypeProgrammatic for edge in data), count)
"""


@pytest.mark.parametrize("switch", ["0", None])
def test_the_switch_reaches_every_kernel(switch: str | None) -> None:
    pytest.importorskip("cuda.bindings.runtime")
    env = {k: v for k, v in os.environ.items() if k != "DIONW_GEMM_PDL"} | {"PYTHONPATH": ROOT}
    if switch is not None:
        env["DIONW_GEMM_PDL"] = switch
    done = subprocess.run([sys.executable, "-c", CHILD], env=env, capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert done.returncode == 0, done.stdout + done.stderr
    programmatic, edges = map(int, done.stdout.split("EDGES")[-1].split())
    assert edges > 5
    assert programmatic == 0 if switch == "0" else programmatic > 0
