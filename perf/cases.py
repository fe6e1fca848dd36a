"""Performance cases: what a user of this package has it do, through its public entry points.

Six kinds of work, each with its range of sizes:

  train      one optimisation step of an MLP (forward, MSE loss, backward, SGD update)
  predict    one serving call: a host batch in, the model's outputs back on the host
  pointwise  an elementwise op under an MSE loss, forward and backward
  reduce     a reduction under an MSE loss, forward and backward
  softmax    softmax cross-entropy written with the package's ops, forward and backward
  matmul     a product under an MSE loss, forward and both gradients

All of it is Float32, the type of every configuration of this repository.
"""

from __future__ import annotations

import math
from types import SimpleNamespace

import torch

import nanotorch_b200 as nt
import nanotorch_b200.nn as nn

UNARY = ("exp", "log", "sqrt", "tanh", "sigmoid", "relu", "neg", "pow")
BINARY = ("add", "sub", "mul", "truediv")
REDUCTIONS = ("sum", "mean", "max", "min")
F32 = 4  # bytes


# ---------------------------------------------------------------------------------------------
# the cases
def listed():
    return [
        # The smallest call there is in earnest: one sample through a trained 784-256-10 classifier.
        {"name": "predict 784-256-10 b1", "kind": "predict", "dims": "784-256-10", "act": "relu", "batch": 1},
        # The small training configuration (Linear-ReLU-Linear, batch 256): some forty small launches a step,
        # issued one by one as a training loop does ...
        {"name": "train 784-256-10 b256", "kind": "train", "dims": "784-256-10", "act": "relu", "batch": 256,
         "lr": 0.01, "graph": False},
        # ... and the same step captured once and replayed, as a loop that minds its launches does.
        {"name": "train 784-256-10 b256 graph", "kind": "train", "dims": "784-256-10", "act": "relu", "batch": 256,
         "lr": 0.01, "graph": True},
        # The large training configuration: 8 x Linear(4096, 4096) with Tanh, the whole global batch on one GPU.
        {"name": "train 8x4096 b16384", "kind": "train", "dims": "-".join(["4096"] * 9), "act": "tanh",
         "batch": 16384, "lr": 0.001, "graph": False},
        # The elementwise sweep's size: a dense binary op with two gradients ...
        {"name": "mul 4096x4096", "kind": "pointwise", "op": "mul", "layout": "dense", "rows": 4096, "cols": 4096},
        # ... one operand seen through a transposed view ...
        {"name": "truediv transposed 4096x4096", "kind": "pointwise", "op": "truediv", "layout": "transposed",
         "rows": 4096, "cols": 4096},
        # ... and an activation at a ragged size between latency and bandwidth.
        {"name": "tanh 1023x1027", "kind": "pointwise", "op": "tanh", "layout": "dense", "rows": 1023, "cols": 1027},
        # The reduction sweep's size, over the strided dimension, with the extremum's masked gradient.
        {"name": "max axis 0 8192x8192", "kind": "reduce", "op": "max", "axis": 0, "rows": 8192, "cols": 8192},
        # A classification loss over a batch of logits: row reductions and column broadcasts.
        {"name": "softmax 4096x1000", "kind": "softmax", "rows": 4096, "cols": 1000},
        # The product configurations: square and batched on the tensor cores (the default mode) ...
        {"name": "matmul 4096x4096x4096", "kind": "matmul", "batch": 1, "m": 4096, "k": 4096, "n": 4096,
         "exact": False},
        {"name": "matmul 32x512x512x512", "kind": "matmul", "batch": 32, "m": 512, "k": 512, "n": 512,
         "exact": False},
        # ... and the rectangular one in the exact Float32 mode.
        {"name": "matmul exact 8192x1024x4096", "kind": "matmul", "batch": 1, "m": 8192, "k": 1024, "n": 4096,
         "exact": True},
    ]


def _size(rng, low, high):
    """A size between low and high, even over its logarithm; one in two is a multiple of 32 where there is room."""
    v = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    if v >= 32 and rng.random() < 0.5:
        v = v // 32 * 32
    return max(low, min(high, v))


def draw(rng):
    kind = rng.choice(("train", "predict", "pointwise", "reduce", "softmax", "matmul"))
    if kind in ("train", "predict"):
        depth = rng.randint(1, 8)
        width = _size(rng, 16, 4096)
        dims = [_size(rng, 16, 4096)] + [width] * (depth - 1) + [_size(rng, 2, 4096)]
        case = {"kind": kind, "dims": "-".join(map(str, dims)), "act": rng.choice(("relu", "tanh")),
                "batch": _size(rng, 1, 16384 if kind == "train" else 256)}
        if kind == "train":
            case.update(lr=rng.choice((0.01, 0.001)), graph=rng.random() < 0.3)
        return case
    if kind == "pointwise":
        op = rng.choice(UNARY + BINARY)
        layout = rng.choice(("dense", "dense", "transposed") if op in UNARY else
                            ("dense", "dense", "row", "column", "transposed"))
        return {"kind": kind, "op": op, "layout": layout, "rows": _size(rng, 1, 8192), "cols": _size(rng, 1, 8192)}
    if kind == "reduce":
        return {"kind": kind, "op": rng.choice(REDUCTIONS), "axis": rng.choice((0, 1, None)),
                "rows": _size(rng, 1, 8192), "cols": _size(rng, 2, 16384)}
    if kind == "softmax":
        return {"kind": kind, "rows": _size(rng, 1, 16384), "cols": _size(rng, 2, 4096)}
    case = {"kind": kind, "batch": rng.choice((1, 1, 1, rng.randint(2, 32))), "m": _size(rng, 16, 4096),
            "k": _size(rng, 16, 4096), "n": _size(rng, 16, 4096), "exact": rng.random() < 0.25}
    while case["batch"] > 1 and work(case)["flops"] > (1e12 if case["exact"] else 8e12):
        case["batch"] //= 2
    return case


def _dims(case):
    return [int(d) for d in case["dims"].split("-")]


# ---------------------------------------------------------------------------------------------
# inputs and outputs
class _DeviceArray:
    """What the CUDA array interface says of a tensor of the package; keeps its storage alive."""

    def __init__(self, t):
        strides, offset = t.strides
        self.owner = t.storage
        self.__cuda_array_interface__ = {
            "shape": t.shape, "strides": tuple(F32 * s for s in strides), "typestr": "<f4", "version": 2,
            "data": (t.storage.data_ptr + F32 * offset, False)}


def _seen(t):
    """A tensor of the package as a torch tensor over the same memory."""
    return torch.as_tensor(_DeviceArray(t), device="cuda")


def _tensor(values, requires_grad=False):
    """A tensor of the package with the values of a torch tensor on the device."""
    storage = nt._C.Storage.allocate(values.numel(), nt.float32, nt.Device.Cuda)
    t = nt.Tensor._new_contiguous(storage, tuple(values.shape))
    torch.cuda.synchronize()
    _seen(t).copy_(values)
    torch.cuda.synchronize()
    if requires_grad:
        t.enable_grad()
    return t


class _Random:
    """Inputs on the device, from a seed."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.gen, device="cuda")

    def uniform(self, low, high, *shape):
        return low + (high - low) * torch.rand(*shape, generator=self.gen, device="cuda")


def _model(case, seed):
    """The layers, initialised on the device from the seed."""
    mode = nt._C.get_rng_mode()
    nt._C.set_rng_mode(nt._C.RNG_DEVICE_PHILOX)
    nt.manual_seed(seed)
    dims = _dims(case)
    layers = []
    for i, (fan_in, fan_out) in enumerate(zip(dims, dims[1:])):
        if i:
            layers.append(nn.ReLU() if case["act"] == "relu" else nn.Tanh())
        layers.append(nn.Linear(fan_in, fan_out, device="cuda"))
    nt._C.set_rng_mode(mode)
    return nn.Sequential(*layers)


def prepare(case, seed):
    rng = _Random(seed)
    s = SimpleNamespace(kind=case["kind"], case=case)
    if s.kind in ("train", "predict"):
        s.model = _model(case, seed)
        dims = _dims(case)
        x = rng.normal(case["batch"], dims[0])
        if s.kind == "predict":
            s.x = x.cpu().numpy()
            return s
        s.x, s.y = _tensor(x), _tensor(rng.normal(case["batch"], dims[-1]))
        s.opt = nn.GradientDescent(s.model.parameters(), lr=case["lr"])
        s.params = [_seen(p) for p in s.model.parameters()]
        if case["graph"]:
            for _ in range(2):  # set-up that must not land in the capture
                _train_step(s)
            s.graph = nt._C.Graph()
            with s.graph.capture():
                s.loss = _train_step(s)
            s.loss_seen = _seen(s.loss)
        return s
    if s.kind == "matmul":
        lead = (case["batch"],) if case["batch"] > 1 else ()
        m, k, n = case["m"], case["k"], case["n"]
        s.a = _tensor(rng.uniform(-1, 1, *lead, m, k), requires_grad=True)
        s.b = _tensor(rng.uniform(-1, 1, *lead, k, n), requires_grad=True)
        s.target = _tensor(rng.normal(*lead, m, n))
        s.mode = nt._C.MATMUL_EXACT_FP32 if case["exact"] else nt._C.MATMUL_3XTF32
        return s
    rows, cols = case["rows"], case["cols"]
    if s.kind == "softmax":
        s.x = _tensor(3 * rng.normal(rows, cols), requires_grad=True)
        labels = torch.randint(cols, (rows,), generator=rng.gen, device="cuda")
        s.labels = _tensor(torch.nn.functional.one_hot(labels, cols).float())
        return s
    if s.kind == "reduce":
        # sums of U(0, 1), the values of the package's own rand; extrema of N(0, 1)
        s.x = _tensor(rng.uniform(0, 1, rows, cols) if case["op"] in ("sum", "mean") else rng.normal(rows, cols),
                      requires_grad=True)
        s.target = _tensor(rng.normal(*{0: (cols,), 1: (rows,), None: ()}[case["axis"]]))
        return s
    op, layout = case["op"], case["layout"]
    positive = op in ("log", "sqrt")  # these on U(0.1, 10), the other unary ops on N(0, 1), binary ones on U(-1, 1)
    dense = (cols, rows) if layout == "transposed" and op in UNARY else (rows, cols)
    s.a = _tensor(rng.uniform(0.1, 10, *dense) if positive else
                  rng.normal(*dense) if op in UNARY else rng.uniform(-1, 1, *dense), requires_grad=True)
    if op in BINARY:
        shape = {"dense": (rows, cols), "row": (cols,), "column": (rows, 1), "transposed": (cols, rows)}[layout]
        s.b = _tensor(rng.uniform(0.5, 2, *shape) if op == "truediv" else rng.uniform(-1, 1, *shape),
                      requires_grad=True)
    s.target = _tensor(rng.normal(rows, cols))
    return s


# ---------------------------------------------------------------------------------------------
# one pass
def _mse(y, target):
    return nt.mean((y - target) ** 2)


def _train_step(s):
    loss = _mse(s.model(s.x), s.y)
    s.opt.zero_grad()
    loss.backward()
    s.opt.step()
    return loss


def _apply(op, a, b):
    if op == "add":
        return a + b
    if op == "sub":
        return a - b
    if op == "mul":
        return a * b
    if op == "truediv":
        return a / b
    if op == "pow":
        return a ** 2.0
    if op == "neg":
        return -a
    return getattr(nt, op)(a)


def _loss_and_grads(loss, *leaves):
    for t in leaves:
        t.zero_grad()
    loss.backward()
    return [_seen(loss)] + [_seen(t.grad) for t in leaves]


def run(s):
    case = s.case
    if s.kind == "predict":
        with nt.no_grad():
            return s.model(nt.Tensor.from_numpy(s.x, "cuda")).numpy()
    if s.kind == "train":
        if case["graph"]:
            s.graph.replay()
            return [s.loss_seen] + s.params
        return [_seen(_train_step(s))] + s.params
    if s.kind == "matmul":
        nt._C.set_matmul_mode(s.mode)
        out = _loss_and_grads(_mse(s.a @ s.b, s.target), s.a, s.b)
        nt._C.set_matmul_mode(nt._C.MATMUL_3XTF32)
        return out
    if s.kind == "softmax":
        e = nt.exp(s.x - s.x.max(axis=1, keepdim=True))
        p = e / e.sum(axis=1, keepdim=True)
        return _loss_and_grads(nt.mean(-(nt.log(p) * s.labels).sum(axis=1)), s.x)
    if s.kind == "reduce":
        return _loss_and_grads(_mse(getattr(s.x, case["op"])(axis=case["axis"]), s.target), s.x)
    op, turned = case["op"], case["layout"] == "transposed"
    if op in UNARY:
        return _loss_and_grads(_mse(_apply(op, s.a.T if turned else s.a, None), s.target), s.a)
    return _loss_and_grads(_mse(_apply(op, s.a, s.b.T if turned else s.b), s.target), s.a, s.b)


# ---------------------------------------------------------------------------------------------
def work(case):
    """What a pass cannot do without: its inputs read once, its outputs written once, its products."""
    kind = case["kind"]
    if kind in ("train", "predict"):
        dims, batch = _dims(case), case["batch"]
        weights = [a * b for a, b in zip(dims, dims[1:])]
        params = sum(weights) + sum(dims[1:])
        io = batch * (dims[0] + dims[-1])
        if kind == "predict":
            return {"bytes": F32 * (params + io), "flops": 2 * batch * sum(weights)}
        # forward, weight gradients, and input gradients of every layer but the first
        return {"bytes": F32 * (2 * params + io), "flops": 2 * batch * (3 * sum(weights) - weights[0])}
    if kind == "matmul":
        b, m, k, n = case["batch"], case["m"], case["k"], case["n"]
        return {"bytes": F32 * b * (2 * m * k + 2 * k * n + m * n), "flops": 6 * b * m * k * n}
    n = case["rows"] * case["cols"]
    if kind == "softmax":
        return {"bytes": F32 * 3 * n, "flops": 8 * n}  # logits, labels in; gradient out
    if kind == "reduce":
        kept = {0: case["cols"], 1: case["rows"], None: 1}[case["axis"]]
        # a sum's gradient is the same along the reduced dimension: one value of each is written
        grad = kept if case["op"] in ("sum", "mean") else n
        return {"bytes": F32 * (n + kept + grad), "flops": 2 * n}
    other = 0 if case["op"] in UNARY else {"row": case["cols"], "column": case["rows"]}.get(case["layout"], n)
    return {"bytes": F32 * (3 * n + 2 * other), "flops": 8 * n}


def tolerance(case):
    """Float32 throughout: sums and products within the order of their additions."""
    return {"rel": 1e-5}
