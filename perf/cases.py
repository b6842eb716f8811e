"""The work this package is timed on: optimizer steps and batched orthogonalizations.

Two paths, both through the public entry points:

* ``step``: ``Dion.step()`` of a routed parameter set in the middle of training
  (momentum, variance and AdamW moments already hold values).  Returns every
  weight and every piece of optimizer state the step updates.
* ``ortho``: ``newton_schulz_fn(kind)(batch, eps)``, the batched polar factor on
  its own, as a caller with its own momentum uses it.

Parameter sets are shapes only (nothing is run forward); gradients are
N(0, 1e-3^2), weights N(0, 0.02^2), as the package's benchmark draws them.
"""

from __future__ import annotations

import math
import random
from typing import Any

import torch
from torch import Tensor, nn

import dionw_b200 as dionw
from dionw_b200 import EMAConfig, MatrixUpdate, MomentumForm, NewtonSchulz, Route, RouteKind, RowNormalization
from dionw_b200.newton_schulz import newton_schulz_fn

Case = dict[str, Any]
DEVICE = torch.device("cuda", 0)
DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}

UPDATES = {
    "dion3": dionw.DION3_UPDATE,
    "muon": dionw.MUON_UPDATE,
    # NorMuon rows on the bf16 Polar Express iteration, every other setting as the default
    "polar": MatrixUpdate(NewtonSchulz.POLAR_EXPRESS, RowNormalization.NORMUON, MomentumForm.HEAVY_BALL),
}

# No drawn case costs more than the largest listed one of its path.
MAX_STEP_PARAMETERS = 900e6
MAX_STEP_FLOPS = 8e12
MAX_ORTHO_COUNT = 16
MAX_ORTHO_SIDES = (4096, 14336)   # the smaller and the larger side of one matrix


def _ortho(name: str, count: int, rows: int, cols: int, dtype: str, kind: str = "gram") -> Case:
    return {"name": name, "path": "ortho", "count": count, "rows": rows, "cols": cols, "dtype": dtype, "kind": kind}


def _step(name: str, style: str, layers: int, width: int, kv: int, ff: int, vocab: int, update: str = "dion3",
          ema: bool = False, weight_decay: float = 0.05) -> Case:
    return {"name": name, "path": "step", "style": style, "layers": layers, "width": width, "kv": kv, "ff": ff,
            "vocab": vocab, "update": update, "ema": ema, "weight_decay": weight_decay}


def listed() -> list[Case]:
    return [
        # One small matrix: a caller that orthogonalizes layer by layer.  Latency of a call.
        _ortho("ortho 1x256x1024 fp32", 1, 256, 1024, "fp32"),
        # The microbenchmark's batches: square (standard iteration), wide, and large.
        _ortho("ortho 16x1024x1024 bf16", 16, 1024, 1024, "bf16"),
        _ortho("ortho 16x1024x4096 bf16", 16, 1024, 4096, "bf16"),
        _ortho("ortho 16x4096x14336 bf16", 16, 4096, 14336, "bf16"),
        # Tall blocks of no round size: iterated transposed.
        _ortho("ortho 6x1531x517 fp32", 6, 1531, 517, "fp32"),
        # The smallest step: one selected matrix and one bias.
        _step("step single 1024x4096", "single", 1, 4096, 1024, 0, 0),
        # A small language model: every matrix below 1024 on one side, so all rows are updated.
        _step("step gpt2-small", "gpt2", 12, 768, 768, 3072, 50257),
        # The same model under the plain Muon settings (Keller iteration, Nesterov, no NorMuon).
        _step("step gpt2-small muon", "gpt2", 12, 768, 768, 3072, 50257, update="muon"),
        # Large language models: layers of two sizes, the default settings; one with a GPU EMA.
        _step("step llama3-8b 4 layers", "llama", 4, 4096, 1024, 14336, 16032),
        _step("step llama3-8b 2 layers ema", "llama", 2, 4096, 1024, 14336, 16032, ema=True),
        _step("step llama3-70b 1 layer", "llama", 1, 8192, 1024, 28672, 16032),
        # An image encoder of no round width: a 4-D patch embedding, a fused projection stepped
        # head group by head group, biases, learned tokens.
        _step("step encoder 1100 wide", "encoder", 6, 1100, 0, 2930, 1000),
    ]


# ---------------------------------------------------------------------------
# drawn cases
# ---------------------------------------------------------------------------
def _spread(rng: random.Random, low: float, high: float) -> float:
    return math.exp(rng.uniform(math.log(low), math.log(high)))


def _size(rng: random.Random, low: float, high: float) -> int:
    """A size of the range: often a multiple of 64 or 8, sometimes any whole number."""
    value = _spread(rng, low, high)
    unit = rng.choice((64, 64, 8, 1))
    return int(min(high, max(low, unit * max(1, round(value / unit)))))


def draw(rng: random.Random) -> Case:
    if rng.random() < 0.5:
        small, large = sorted((_size(rng, 64, MAX_ORTHO_SIDES[0]), _size(rng, 64, MAX_ORTHO_SIDES[1])))
        small = min(small, MAX_ORTHO_SIDES[0])
        if rng.random() < 0.15:
            large = small
        rows, cols = (large, small) if rng.random() < 0.3 else (small, large)
        case = _ortho("", max(1, int(_spread(rng, 1, MAX_ORTHO_COUNT + 1))), rows, cols, rng.choice(tuple(DTYPES)),
                      rng.choice(("gram", "gram", "gram", "polar_express", "keller")))
    else:
        while True:
            style = rng.choice(("llama", "llama", "gpt2", "encoder", "single"))
            width = _size(rng, 192, 6144)
            kv = max(8, width // rng.choice((1, 2, 4, 8)))
            unit = rng.choice((64, 8, 2))
            ff = unit * max(1, int(width * rng.uniform(2.0, 4.0) / unit))
            case = _step("", style, rng.randint(1, 4 if style == "llama" else 12), width, kv, ff,
                         _size(rng, 1000, 50000), rng.choice(("dion3", "dion3", "dion3", "muon", "polar")),
                         style == "llama" and rng.random() < 0.3, rng.choice((0.0, 0.05, 0.1)))
            shapes = _shapes(case)
            if (sum(math.prod(s) for _, s in shapes) <= MAX_STEP_PARAMETERS
                    and sum(f for *_, f in _matrices(case)) <= MAX_STEP_FLOPS):
                break
    del case["name"]
    return case


# ---------------------------------------------------------------------------
# parameter sets
# ---------------------------------------------------------------------------
def _shapes(case: Case) -> list[tuple[str, tuple[int, ...]]]:
    """``(name, shape)`` of every parameter, in registration order."""
    d, kv, ff, vocab = case["width"], case["kv"], case["ff"], case["vocab"]
    style = case["style"]
    if style == "single":
        return [("weight", (max(64, d // 4), d)), ("bias", (d,))]
    out: list[tuple[str, tuple[int, ...]]] = []
    if style == "llama":
        out.append(("embed", (vocab, d)))
        for i in range(case["layers"]):
            out += [(f"{i}.q", (d, d)), (f"{i}.k", (kv, d)), (f"{i}.v", (kv, d)), (f"{i}.o", (d, d)),
                    (f"{i}.gate", (ff, d)), (f"{i}.up", (ff, d)), (f"{i}.down", (d, ff)),
                    (f"{i}.norm1", (d,)), (f"{i}.norm2", (d,))]
        return out + [("norm", (d,)), ("lm_head", (vocab, d))]
    if style == "gpt2":
        out += [("embed", (vocab, d)), ("wpe_embed", (1024, d))]
        for i in range(case["layers"]):
            out += [(f"{i}.ln1_w", (d,)), (f"{i}.ln1_b", (d,)), (f"{i}.ln2_w", (d,)), (f"{i}.ln2_b", (d,)),
                    (f"{i}.c_attn", (d, 3 * d)), (f"{i}.c_proj", (d, d)), (f"{i}.fc", (d, ff)), (f"{i}.proj", (ff, d))]
        return out + [("norm", (d,)), ("ln_f_b", (d,))]
    # encoder
    out += [("patch", (d, 3, 16, 16)), ("patch_bias", (d,)), ("cls_token", (1, 1, d)), ("pos_embed", (1, 197, d))]
    for i in range(case["layers"]):
        out += [(f"{i}.norm1", (d,)), (f"{i}.qkv", (3 * d, d)), (f"{i}.qkv_bias", (3 * d,)), (f"{i}.out", (d, d)),
                (f"{i}.norm2", (d,)), (f"{i}.fc1", (ff, d)), (f"{i}.fc1_bias", (ff,)), (f"{i}.fc2", (d, ff)),
                (f"{i}.fc2_bias", (d,))]
    return out + [("norm", (d,)), ("head", (vocab, d)), ("head_bias", (vocab,))]


def _is_table(name: str) -> bool:
    """Parameters that go to AdamW although they are matrices."""
    return name in ("embed", "wpe_embed", "lm_head", "cls_token", "pos_embed")


def _heads(name: str) -> int:
    """Blocks the rows of a fused projection are split into."""
    return 3 if name.endswith(".qkv") else 1


def _matrices(case: Case) -> list[tuple[int, int, int, int, float]]:
    """``(blocks, rows, selected rows, cols, Newton-Schulz FLOPs)`` of every matrix parameter."""
    out = []
    for name, shape in _shapes(case):
        if len(shape) < 2 or _is_table(name):
            continue
        heads = _heads(name)
        rows, cols = shape[0] // heads, math.prod(shape[1:])
        selecting = case["update"] != "muon" and min(rows, cols) >= 1024
        k = math.ceil(0.25 * rows) if selecting else rows
        out.append((heads, rows, k, cols, heads * _orthogonalize_flops(k, cols, case["update"] == "dion3")))
    return out


def _orthogonalize_flops(rows: int, cols: int, gram: bool) -> float:
    """FLOPs of five quintic steps with every symmetric product counted as the half it needs: on the
    ``m x m`` Gram matrix (``3 m^2 n + 7 m^3`` multiply-adds) or on the operand itself, whichever is less."""
    m, n = min(rows, cols), max(rows, cols)
    direct = 2.0 * 5 * (1.5 * m * m * n + 0.5 * m**3)
    return min(direct, 2.0 * (3.0 * m * m * n + 7.0 * m**3)) if gram else direct


class _Flat:
    """One flat fp32 buffer with a view per shape, each on a 512-byte boundary."""

    def __init__(self, shapes: list[tuple[int, ...]]) -> None:
        starts, total = [], 0
        for shape in shapes:
            starts.append(total)
            total += -(-math.prod(shape) // 128) * 128
        self.buffer = torch.zeros(total, device=DEVICE)
        self.views = [self.buffer[s:s + math.prod(shape)].view(shape) for s, shape in zip(starts, shapes)]


class _ParameterSet(nn.Module):
    def __init__(self, names: list[str], values: list[Tensor]) -> None:
        super().__init__()
        self.order = [nn.Parameter(value) for value in values]
        for name, parameter in zip(names, self.order):
            self.register_parameter(name.replace(".", "_"), parameter)


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def prepare(case: Case, seed: int) -> dict[str, Any]:
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    if case["path"] == "ortho":
        x = torch.randn(case["count"], case["rows"], case["cols"], device=DEVICE, generator=gen)
        x /= torch.linalg.vector_norm(x, dim=(1, 2), keepdim=True)   # the microbenchmark's unit Frobenius norm
        return {"call": newton_schulz_fn(NewtonSchulz(case["kind"])), "x": x.to(DTYPES[case["dtype"]])}

    names = [name for name, _ in _shapes(case)]
    shapes = [shape for _, shape in _shapes(case)]
    weights, grads = _Flat(shapes), _Flat(shapes)
    weights.buffer.normal_(0.0, 0.02, generator=gen)
    grads.buffer.normal_(0.0, 1e-3, generator=gen)
    model = _ParameterSet(names, weights.views)
    routes = {}
    for name, parameter, grad in zip(names, model.order, grads.views):
        parameter.grad = grad
        if _is_table(name):
            routes[parameter] = Route(RouteKind.ADAMW)
        elif _heads(name) > 1:
            routes[parameter] = Route(RouteKind.MATRIX, num_heads=_heads(name))
    groups, _ = dionw.param_groups(model, routes=routes, **({"fraction": 1.0} if case["update"] == "muon" else {}))
    optimizer = dionw.Dion(groups, lr=3e-4, weight_decay=case["weight_decay"], matrix_update=UPDATES[case["update"]],
                           ema=EMAConfig(decay=0.9999) if case["ema"] else None)
    # The state of a run that is under way.  AdamW's moments lie in flat buffers, as the weights do;
    # momentum and variance are the optimizer's own slabs, one per shape.
    slabs: dict[int, Tensor] = {}
    adamw = []
    for parameter in model.order:
        optimizer.initialize_state(parameter)
        entry = optimizer.state[parameter]
        if "momentum" not in entry:
            adamw.append(parameter)
            continue
        entry["momentum"].normal_(0.0, 5e-3, generator=gen)
        entry["variance"].uniform_(0.5, 1.2, generator=gen).div_(max(parameter.shape[0], parameter[0].numel()))
        for key in ("momentum", "variance"):
            storage = entry[key].untyped_storage()
            slabs.setdefault(storage.data_ptr(), torch.empty(0, device=DEVICE).set_(storage))
    exp_avg, exp_avg_sq = _Flat([p.shape for p in adamw]), _Flat([p.shape for p in adamw])
    exp_avg.buffer.normal_(0.0, 3e-4, generator=gen)
    exp_avg_sq.buffer.uniform_(0.5e-6, 1.5e-6, generator=gen)
    steps = torch.full((len(adamw),), 1000.0, device=DEVICE)
    for i, parameter in enumerate(adamw):
        optimizer.state[parameter].update(exp_avg=exp_avg.views[i], exp_avg_sq=exp_avg_sq.views[i],
                                          adamw_step=steps[i])
    return {"optimizer": optimizer, "model": model, "ema": case["ema"],
            "outputs": {"weights": weights.buffer, "slabs": list(slabs.values()), "exp_avg": exp_avg.buffer,
                        "exp_avg_sq": exp_avg_sq.buffer, "steps": steps}}


def run(state: dict[str, Any]) -> Any:
    if "call" in state:
        return state["call"](state["x"], 1e-8)
    optimizer = state["optimizer"]
    optimizer.step()
    outputs = state["outputs"]
    if state["ema"]:
        outputs = {**outputs, "shadows": [optimizer.state[p]["ema_shadow"] for p in state["model"].order]}
    return outputs


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case: Case) -> dict[str, float]:
    if case["path"] == "ortho":
        elements = case["count"] * case["rows"] * case["cols"]
        flops = case["count"] * _orthogonalize_flops(case["rows"], case["cols"], case["kind"] == "gram")
        return {"bytes": elements * (DTYPES[case["dtype"]].itemsize + 2.0), "flops": flops}
    everything = sum(math.prod(shape) for _, shape in _shapes(case))
    matrices = _matrices(case)
    matrix_elements = sum(blocks * rows * cols for blocks, rows, _, cols, _ in matrices)
    # matrices: gradient read, momentum and weight read and written; AdamW: weight and both moments
    # read and written, gradient read; the EMA reads and writes its shadow
    moved = 20.0 * matrix_elements + 28.0 * (everything - matrix_elements) + (8.0 * everything if case["ema"] else 0.0)
    return {"bytes": moved, "flops": sum(f for *_, f in matrices)}


def tolerance(case: Case) -> Any:
    """About four times the distance of two correct evaluations on a B200: the Gram products mirrored
    against computed in full (2.9e-3 on the result, at most 1.4e-2 on an element; 1.6e-4 and 1.8e-3 on
    the variance a step leaves), the bf16 iterations of an input scaled by 1.0003 (1.0e-2, 7.7e-2),
    each as far from the fp64 polynomial as from one another."""
    bf16_iteration = case["kind"] != "gram" if case["path"] == "ortho" else case["update"] != "dion3"
    if case["path"] == "ortho":
        return {"rel": 3e-2, "max": 0.3} if bf16_iteration else {"rel": 1e-2, "max": 6e-2}
    return {"rel": 3e-3, "max": 3e-2} if bf16_iteration else {"rel": 8e-4, "max": 1e-2}


# ---------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------
_S = 1.05   # safety factor the Gram iteration divides its coefficients by, to the first, third and fifth power
_GRAM = [(8.28721201814563 / _S, -23.595886519098837 / _S**3, 17.300387312530933 / _S**5),
         (4.107059111542203 / _S, -2.9478499167379106 / _S**3, 0.5448431082926601 / _S**5),
         (3.9486908534822946 / _S, -2.908902115962949 / _S**3, 0.5518191394370137 / _S**5),
         (3.3184196573706015 / _S, -2.488488024314874 / _S**3, 0.51004894012372 / _S**5),
         (2.300652019954817 / _S, -1.6689039845747493 / _S**3, 0.4188073119525673 / _S**5)]
_POLAR = [(8.156554524902461, -22.48329292557795, 15.878769915207462),
          (4.042929935166739, -2.808917465908714, 0.5000178451051316),
          (3.8916678022926607, -2.772484153217685, 0.5060648178503393),
          (3.285753657755655, -2.3681294933425376, 0.46449024233003106),
          (2.3465413258596377, -1.7097828382687081, 0.42323551169305323)]
# kind -> the five steps' coefficients and the factor on the Frobenius norm
_ITERATIONS = {"gram": (_GRAM, 1.0), "polar_express": (_POLAR, 1.02), "keller": ([(3.4445, -4.7750, 2.0315)] * 5, 1.0)}
MAX_EXACT_FLOPS = 1e14   # a few seconds of 64-bit products


def _polar(matrix: Tensor, kind: str, epsilon: float = 1e-8) -> Tensor:
    """The five-step polynomial of one matrix."""
    if matrix.shape[0] > matrix.shape[1]:
        return _polar(matrix.T, kind, epsilon).T
    table, norm_scale = _ITERATIONS[kind]
    x = matrix.double()
    x = x / (x.norm() * norm_scale + epsilon)
    for a, b, c in table:
        gram = x @ x.T
        x = a * x + (b * gram + c * (gram @ gram)) @ x
    return x


def exact(case: Case, seed: int) -> Any:
    """What ``run`` returns for ``prepare(case, seed)``, in 64 bits; None where that takes too long."""
    if case["path"] == "ortho":
        small, large = sorted((case["rows"], case["cols"]))
        if case["count"] * 20.0 * (small * small * large + small**3 / 2) > MAX_EXACT_FLOPS:
            return None
        x = prepare(case, seed)["x"]
        return torch.stack([_polar(matrix, case["kind"]) for matrix in x])
    cost = sum(blocks * 20.0 * (min(k, cols) ** 2 * max(k, cols) + min(k, cols) ** 3 / 2)
               for blocks, _, k, cols, _ in _matrices(case))
    if cost > MAX_EXACT_FLOPS:
        return None
    state = prepare(case, seed)
    optimizer, outputs = state["optimizer"], state["outputs"]
    # every buffer that holds results, by its address, as a 64-bit copy the results are written to
    copies = {}
    for buffer in (outputs["weights"], *outputs["slabs"], outputs["exp_avg"], outputs["exp_avg_sq"], outputs["steps"]):
        copies[buffer.untyped_storage().data_ptr()] = buffer.double()

    def at(tensor: Tensor) -> Tensor:
        copy = copies[tensor.untyped_storage().data_ptr()]
        return copy.as_strided(tensor.shape, tensor.stride(), tensor.storage_offset())

    settings = {id(p): group for group in optimizer.param_groups for p in group["params"]}
    kind = {"dion3": "gram", "muon": "keller", "polar": "polar_express"}[case["update"]]
    nesterov, normuon = case["update"] == "muon", case["update"] != "muon"
    matrices = iter(_matrices(case))
    names = [name for name, shape in _shapes(case)]
    for name, parameter in zip(names, state["model"].order):
        group, entry = settings[id(parameter)], optimizer.state[parameter]
        lr, decay = group["lr"], group["weight_decay"]
        weight, grad = at(parameter), parameter.grad.double()
        weight *= 1.0 - lr * decay
        if parameter.ndim < 2 or _is_table(name):
            beta1, beta2 = group["betas"]
            mean, square, step = at(entry["exp_avg"]), at(entry["exp_avg_sq"]), at(entry["adamw_step"])
            step += 1.0
            mean.mul_(beta1).add_(grad, alpha=1.0 - beta1)
            square.mul_(beta2).add_(grad * grad, alpha=1.0 - beta2)
            root = square.sqrt() / math.sqrt(1.0 - beta2 ** float(step)) + group["eps"]
            weight -= lr / (1.0 - beta1 ** float(step)) * mean / root
            continue
        blocks, rows, k, cols, _ = next(matrices)
        size = -lr * 0.2 * math.sqrt(max(rows, cols)) * math.sqrt(min(rows, cols) / min(k, cols))
        momentum = at(entry["momentum"]).view(blocks, rows, cols)
        variance = at(entry["variance"]).view(blocks, rows)
        momentum += grad.view(blocks, rows, cols)
        for m, v, w, g in zip(momentum, variance, weight.view(blocks, rows, cols), grad.view(blocks, rows, cols)):
            chosen = m.abs().sum(1).topk(k).indices if k < rows else torch.arange(rows, device=DEVICE)
            source = m[chosen]
            m[chosen] = group["momentum"] * source
            update = _polar(group["momentum"] * source + g if nesterov else source, kind)
            if normuon:
                squares = (update * update).sum(1)
                v[chosen] = torch.lerp(v[chosen], squares / cols, 1.0 - group["muon_beta2"])
                divisor = v[chosen].sqrt() + 1e-8
                update = update / divisor[:, None] * (squares.sum().sqrt() / (squares / divisor**2).sum().sqrt())
            w[chosen] += size * update
    result: dict[str, Any] = {
        "weights": at(outputs["weights"]), "slabs": [at(slab) for slab in outputs["slabs"]],
        "exp_avg": at(outputs["exp_avg"]), "exp_avg_sq": at(outputs["exp_avg_sq"]), "steps": at(outputs["steps"])}
    if case["ema"]:
        result["shadows"] = [at(p).clone() for p in state["model"].order]   # the first update copies the weights
    return result
