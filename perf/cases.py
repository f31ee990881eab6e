"""
Performance cases: the work a program does through the public API, over the
range of sizes that programs use.

Each kind of case is one family of entry points:

  elementwise  array operators, math methods, broadcasting, a fused chain
  reduce       sum / mean / maximum / minimum / prod / argmax over every axis
  gather       flat gather by uint32 indices, row gather (minibatches)
  prng         Xoshiro128pp uniform, normal and raw outputs
  matmul       ``vk.matmul`` in its three precisions (a vector operand too)
  dense        one Dense layer on torch tensors, forward and backward
  mlp          one ``Sequence.train`` step (Adam), eager or as a graph
  grouped      one ``GroupedSequence.train`` step of uneven models (SGD)

Inputs are drawn by torch from the seed and uploaded through ``Array``.
``run`` returns the arrays of a pass; they become torch tensors (views of the
same device memory) only where somebody looks at them, since a program that
goes on computing on the device makes no such views.
"""
import math

import numpy as np
import torch

import vulkpy_gb300 as vk
from vulkpy_gb300 import autograd, nn

_F32_1EM3 = float(np.float32(1e-3))
_LR = 1e-4  # the widest of the grouped models still converges with it


def listed():
    return [
        # the small op suite: launch latency and host cost per call decide
        {"name": "elementwise_small", "kind": "elementwise", "rows": 512, "cols": 1024},
        # the bandwidth suite's matrix, 1 GiB: device memory bandwidth decides
        {"name": "elementwise_large", "kind": "elementwise", "rows": 8192, "cols": 32768},
        # statistics of a small batch of odd-sized images or sequences
        {"name": "reduce_ragged", "kind": "reduce", "d0": 37, "d1": 257, "d2": 129},
        # statistics of a whole data set held on the device
        {"name": "reduce_large", "kind": "reduce", "d0": 1, "d1": 8192, "d2": 32768},
        # lookups by random index in a table larger than the L2 cache
        {"name": "gather_large", "kind": "gather", "rows": 8192, "cols": 32768, "n_idx": 1 << 26, "axis": -1},
        # simulation inputs: many generator states, long streams
        {"name": "prng_large", "kind": "prng", "states": 1 << 20, "n": 1 << 27},
        # a user's ``a @ b`` as it comes: default precision, no round sizes
        {"name": "matmul_fp32_ragged", "kind": "matmul", "m": 1000, "k": 1531, "n": 777, "precision": "fp32"},
        # large products, the precision chosen by the caller
        {"name": "matmul_bf16x3_large", "kind": "matmul", "m": 4096, "k": 4096, "n": 4096, "precision": "bf16x3"},
        {"name": "matmul_bf16_large", "kind": "matmul", "m": 8192, "k": 8192, "n": 8192, "precision": "bf16"},
        # a layer of a torch program, default precision, forward and backward
        {"name": "dense_fp32", "kind": "dense", "batch": 256, "n_in": 784, "n_out": 1024, "act": "sigmoid",
         "precision": "fp32"},
        # training a digit classifier: the step captured once and replayed
        {"name": "mlp_graph", "kind": "mlp", "batch": 256, "n_in": 784, "hidden": 1024, "n_out": 10,
         "precision": "bf16x3", "compiled": True},
        # a sweep of 64 small regressors of uneven sizes, trained together
        {"name": "grouped_graph", "kind": "grouped", "models": 64, "precision": "bf16x3", "sizes": 2},
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["elementwise", "reduce", "gather", "prng", "matmul", "matmul", "dense", "mlp", "grouped"])
    if kind == "elementwise":
        return {"kind": kind, "rows": _log(rng, 8, 8192), "cols": _log(rng, 8, 32768)}
    if kind == "reduce":
        d1, d2 = _log(rng, 8, 8192), _log(rng, 8, 32768)
        return {"kind": kind, "d0": _log(rng, 1, max(1, min(64, (1 << 28) // (d1 * d2)))), "d1": d1, "d2": d2}
    if kind == "gather":
        if rng.random() < 0.5:
            return {"kind": kind, "rows": _log(rng, 8, 8192), "cols": _log(rng, 8, 32768),
                    "n_idx": _log(rng, 32, 1 << 26), "axis": -1}
        return {"kind": kind, "rows": _log(rng, 120, 70000), "cols": _log(rng, 4, 1024),
                "n_idx": _log(rng, 32, 70000), "axis": 0}
    if kind == "prng":
        return {"kind": kind, "states": _log(rng, 64, 1 << 20), "n": _log(rng, 1024, 1 << 27)}
    if kind == "matmul":
        case = {"kind": kind, "m": _log(rng, 16, 8192), "k": _log(rng, 16, 8192), "n": _log(rng, 16, 8192),
                "precision": rng.choice(["fp32", "fp32", "bf16x3", "bf16"])}
        if rng.random() < 0.15:
            case["m"] = 1
        if case["precision"] == "fp32":  # costs no more than the largest bf16 product
            while case["m"] * case["k"] * case["n"] > 1 << 34:
                case[rng.choice("mkn")] = _log(rng, 16, 2048)
        return case
    if kind == "dense":
        return {"kind": kind, "batch": _log(rng, 8, 4096), "n_in": _log(rng, 16, 2048), "n_out": _log(rng, 10, 2048),
                "act": rng.choice(["sigmoid", "none"]), "precision": rng.choice(["fp32", "fp32", "bf16x3"])}
    if kind == "mlp":
        return {"kind": kind, "batch": _log(rng, 32, 512), "n_in": _log(rng, 4, 1024), "hidden": _log(rng, 32, 1024),
                "n_out": _log(rng, 3, 10), "precision": rng.choice(["fp32", "bf16x3"]),
                "compiled": rng.random() < 0.5}
    return {"kind": "grouped", "models": _log(rng, 2, 64), "precision": rng.choice(["fp32", "bf16x3"]),
            "sizes": rng.randrange(1 << 20)}


# ------------------------------------------------------------------ inputs


def _torch_rng(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, *shape):
    return torch.randn(shape, generator=g, device="cuda")


def _uniform(g, lo, hi, *shape):
    return torch.rand(shape, generator=g, device="cuda") * (hi - lo) + lo


def _array(gpu, t):
    return vk.Array(gpu, data=t.cpu().numpy())


class _Device:
    """The device memory of an Array, for torch (uint32 seen as int32)."""

    def __init__(self, a):
        self.array = a
        kind = "<i4" if isinstance(a, vk.U32Array) else "<f4"
        self.__cuda_array_interface__ = {"shape": tuple(a.shape), "typestr": kind, "data": (a._buf.ptr, False),
                                         "version": 3}


def _tensor(v):
    if isinstance(v, (list, tuple)):  # one kind of output of several models
        return torch.cat([_tensor(a).reshape(-1) for a in v])
    return v if isinstance(v, torch.Tensor) else torch.as_tensor(_Device(v), device="cuda")


class _Outputs(dict):
    """A pass's arrays by name; looking one up gives it as a tensor."""

    def __getitem__(self, key):
        return _tensor(dict.__getitem__(self, key))


def _inputs(case, seed):
    """The case's input tensors (float32 on the GPU; indices int64)."""
    g, kind = _torch_rng(seed), case["kind"]
    if kind == "elementwise":
        r, c = case["rows"], case["cols"]
        return {"x": _normal(g, r, c), "row": _uniform(g, 0.5, 2.0, 1, c), "col": _uniform(g, 0.5, 2.0, r, 1)}
    if kind == "reduce":
        shape = [case["d1"], case["d2"]] if case["d0"] == 1 else [case["d0"], case["d1"], case["d2"]]
        x = _normal(g, *shape)
        return {"x": x, "e": torch.exp(x * 1e-4)}
    if kind == "gather":
        r, c = case["rows"], case["cols"]
        top = r * c if case["axis"] < 0 else r
        return {"x": _normal(g, r, c), "idx": torch.randint(0, top, (case["n_idx"],), generator=g, device="cuda")}
    if kind == "matmul":
        a = (case["k"],) if case["m"] == 1 else (case["m"], case["k"])
        return {"a": _normal(g, *a), "b": _normal(g, case["k"], case["n"])}
    if kind == "dense":
        b, i, o = case["batch"], case["n_in"], case["n_out"]
        return {"x": _normal(g, b, i), "w": _normal(g, o, i) * math.sqrt(2.0 / i), "b": _normal(g, o) * 0.1,
                "dy": _normal(g, b, o) / b}
    if kind == "mlp":
        b, i, h, o = case["batch"], case["n_in"], case["hidden"], case["n_out"]
        y = torch.zeros(b, o, device="cuda")
        y[torch.arange(b, device="cuda"), torch.randint(0, o, (b,), generator=g, device="cuda")] = 1.0
        return {"x": _normal(g, b, i), "y": y,
                "w": [_normal(g, m, n) * math.sqrt(2.0 / n) for m, n in ((h, i), (h, h), (o, h))]}
    if kind == "grouped":
        models = []
        for i, h, o, b in _dims(case):
            models.append({"x": _normal(g, b, i), "y": _normal(g, b, o),
                           "w": [_normal(g, m, n) * math.sqrt(2.0 / n) for m, n in ((h, i), (o, h))]})
        return {"models": models}
    raise ValueError(kind)


def _dims(case):
    """Widths and batch sizes of the grouped models: part of the case, not of
    its values."""
    r = np.random.default_rng(case["sizes"])
    return [(int(r.integers(17, 1022)), int(r.integers(32, 2049)), int(r.integers(2, 65)), int(r.integers(1, 513)))
            for _ in range(case["models"])]


@vk.fusion.fuse
def _chain(x, z):
    t = x * 1.5 + z
    t = t.tanh().exp()
    return t.max(0.5) - z


def _given(w):
    return lambda gpu, shape: _array(gpu, w)


def prepare(case, seed):
    kind, gpu = case["kind"], vk.GPU()
    s = {"kind": kind, "gpu": gpu, "case": case}
    if kind == "prng":
        s["rng"] = vk.random.Xoshiro128pp(gpu, size=case["states"], seed=int(seed))
        return s
    t = _inputs(case, seed)
    if kind in ("elementwise", "reduce", "matmul"):
        s.update({k: _array(gpu, v) for k, v in t.items()})
    elif kind == "gather":
        s.update(x=_array(gpu, t["x"]), idx=vk.U32Array(gpu, data=t["idx"].cpu().numpy().astype(np.uint32)))
    elif kind == "dense":
        s.update({k: v.requires_grad_(k != "dy") for k, v in t.items()})
    elif kind == "mlp":
        gpu.matmul_precision = case["precision"]
        opt = nn.Adam(gpu, lr=1e-3)
        dims = [case["n_in"], case["hidden"], case["hidden"], case["n_out"]]
        d = [nn.Dense(gpu, dims[k], dims[k + 1], w_opt=opt, b_opt=opt, w_init=_given(t["w"][k])) for k in range(3)]
        net = nn.Sequence([d[0], nn.ReLU(), d[1], nn.Sigmoid(), d[2]], nn.SoftmaxCrossEntropyLoss())
        s.update(net=net, dense=d, x=_array(gpu, t["x"]), y=_array(gpu, t["y"]))
        net.train(s["x"], s["y"])
        s["step"] = net.compile(s["x"], s["y"]) if case["compiled"] else lambda: net.train(s["x"], s["y"])
    elif kind == "grouped":
        gpu.matmul_precision = case["precision"]
        nets = []
        for m in t["models"]:
            opt = nn.SGD(lr=_LR)
            d = [nn.Dense(gpu, w.shape[1], w.shape[0], w_opt=opt, b_opt=opt, w_init=_given(w)) for w in m["w"]]
            nets.append(nn.Sequence([d[0], nn.ReLU(), d[1]], nn.MSELoss()))
        group = nn.GroupedSequence(nets)
        xs, ys = [_array(gpu, m["x"]) for m in t["models"]], [_array(gpu, m["y"]) for m in t["models"]]
        group.train(xs, ys)
        graph = vk.graph.Graph(gpu)
        with graph:
            preds, losses = group.train(xs, ys)
        s.update(nets=nets, group=group, xs=xs, ys=ys, graph=graph, preds=preds, losses=losses)
    return s


# --------------------------------------------------------------------- run


def run(state):
    return _Outputs(_RUN[state["kind"]](state))


def _run_elementwise(s):
    x, row, col = s["x"], s["row"], s["col"]
    z = x.abs()
    z += 1e-3
    y = x - col
    y *= row
    return {"add": x + row, "mul": x * col, "div": x / row, "z": z, "pow": z ** col, "sqrt": z.sqrt(), "log": z.log(),
            "exp": x.exp(), "tanh": x.tanh(), "clamp": x.clamp(-0.5, 0.5), "max": x.max(row), "y": y,
            "square": x ** 2.0, "same": x * z, "chain": _chain(x, z)}


def _run_reduce(s):
    x, e = s["x"], s["e"]
    out = {"mean": x.mean(axis=0), "minimum": x.minimum(axis=len(x.shape) - 1),
           "argmax": x.argmax(axis=len(x.shape) - 1), "argmin": x.argmin()}
    for axis in [None] + list(range(len(x.shape))):
        out["sum%s" % axis] = x.sum(axis=axis)
        out["maximum%s" % axis] = x.maximum(axis=axis)
        out["prod%s" % axis] = e.prod(axis=axis)
    return out


def _run_gather(s):
    return {"values": s["x"].gather(s["idx"], axis=None if s["case"]["axis"] < 0 else 0)}


def _run_prng(s):
    shape = (s["case"]["n"],)
    return {"uniform": s["rng"].random(shape=shape), "normal": s["rng"].normal(shape=shape),
            "uint32": s["rng"].randint(shape=shape)}


def _run_matmul(s):
    return {"c": vk.vkarray.matmul(s["a"], s["b"], s["case"]["precision"])}


def _run_dense(s):
    y = autograd.dense(s["x"], s["w"], s["b"], act=s["case"]["act"], precision=s["case"]["precision"])
    dx, dw, db = torch.autograd.grad(y, (s["x"], s["w"], s["b"]), s["dy"])
    return {"y": y, "dx": dx, "dw": dw, "db": db}


def _run_mlp(s):
    pred, loss = s["step"]()
    out = {"pred": pred, "loss": loss}
    for k, d in enumerate(s["dense"]):
        out.update({"w%d" % k: d.w.value, "b%d" % k: d.b.value, "dw%d" % k: d.w.grad, "db%d" % k: d.b.grad})
    return out


def _run_grouped(s):
    s["graph"].launch()
    out = {"pred": s["preds"], "loss": s["losses"]}
    for k in (0, 2):
        layers = [n.L[k] for n in s["nets"]]
        out.update({"w%d" % k: [d.w.value for d in layers], "b%d" % k: [d.b.value for d in layers],
                    "dw%d" % k: [d.w.grad for d in layers], "db%d" % k: [d.b.grad for d in layers]})
    return out


_RUN = {"elementwise": _run_elementwise, "reduce": _run_reduce, "gather": _run_gather, "prng": _run_prng,
        "matmul": _run_matmul, "dense": _run_dense, "mlp": _run_mlp, "grouped": _run_grouped}


# -------------------------------------------------------------------- work


def work(case):
    """Bytes (every call's inputs read once, its outputs written once) and
    operations of one pass."""
    kind = case["kind"]
    if kind == "elementwise":
        n, r, c = case["rows"] * case["cols"], case["rows"], case["cols"]
        # 15 calls of one matrix in and one out, one of two in and one out
        # (the chain and x * z), the row and column operands
        return {"bytes": 4 * (2 * 15 * n + 2 * 3 * n + 4 * c + 3 * r), "flops": 21 * n}
    if kind == "reduce":
        n, dims = case["d0"] * case["d1"] * case["d2"], [d for d in (case["d0"], case["d1"], case["d2"]) if d > 1]
        outs = 3 * (1 + sum(n // d for d in dims)) + n // dims[0] + 2 * (n // dims[-1]) + 1
        calls = 4 + 3 * (1 + len(dims))
        return {"bytes": 4 * (calls * n + outs), "flops": calls * n}
    if kind == "gather":
        width = 1 if case["axis"] < 0 else case["cols"]
        return {"bytes": 4 * case["n_idx"] * (1 + 2 * width), "flops": 0}
    if kind == "prng":
        return {"bytes": 3 * (4 * case["n"] + 32 * min(case["states"], case["n"])), "flops": 60 * case["n"]}
    if kind == "matmul":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": 4 * (m * k + k * n + m * n), "flops": 2 * m * k * n}
    if kind == "dense":
        b, i, o = case["batch"], case["n_in"], case["n_out"]
        # forward: x, w, b -> y; backward: dy, y, x, w -> dx, dw, db
        return {"bytes": 4 * (3 * b * i + 3 * b * o + 3 * o * i + 2 * o), "flops": 6 * b * i * o}
    if kind == "mlp":
        b, i, h, o = case["batch"], case["n_in"], case["hidden"], case["n_out"]
        params = i * h + h + h * h + h + h * o + o
        # the batch, and per parameter value, gradient and both Adam moments
        # read, gradient, value and moments written
        return {"bytes": 4 * (b * (i + 2 * o) + 8 * params), "flops": 6 * b * (i * h + h * h + h * o)}
    total = {"bytes": 0, "flops": 0}
    for i, h, o, b in _dims(case):
        params = i * h + h + h * o + o
        total["bytes"] += 4 * (b * (i + 3 * o) + 3 * params)
        total["flops"] += 6 * b * (i * h + h * o)
    return total


# ------------------------------------------------------------------- exact


def exact(case, seed):
    kind = case["kind"]
    if kind == "prng":
        return _exact_prng(case, seed)
    t = _inputs(case, seed)
    return _EXACT[kind](case, t)


def _exact_elementwise(case, t):
    x, row, col = (t[k].double() for k in ("x", "row", "col"))
    z = x.abs() + _F32_1EM3
    return {"add": x + row, "mul": x * col, "div": x / row, "z": z, "pow": z ** col, "sqrt": z.sqrt(), "log": z.log(),
            "exp": x.exp(), "tanh": x.tanh(), "clamp": x.clamp(-0.5, 0.5), "max": torch.maximum(x, row),
            "y": (x - col) * row, "square": x * x, "same": x * z,
            "chain": torch.exp(torch.tanh(x * 1.5 + z)).clamp(min=0.5) - z}


def _exact_reduce(case, t):
    x, e = t["x"].double(), t["e"].double()
    last = x.dim() - 1
    out = {"mean": x.mean(0), "minimum": x.amin(last), "argmax": None, "argmin": None,
           "sumNone": x.sum().reshape(1), "maximumNone": x.max().reshape(1), "prodNone": e.prod().reshape(1)}
    for a in range(x.dim()):
        out.update({"sum%d" % a: x.sum(a), "maximum%d" % a: x.amax(a), "prod%d" % a: e.prod(a)})
    return out


def _exact_gather(case, t):
    x = t["x"].double()
    return {"values": x.reshape(-1)[t["idx"]] if case["axis"] < 0 else x[t["idx"]]}


def _exact_matmul(case, t):
    return {"c": t["a"].double() @ t["b"].double()}


def _exact_dense(case, t):
    x, w, b, dy = (t[k].double() for k in ("x", "w", "b", "dy"))
    y = x @ w.T + b
    g = dy
    if case["act"] == "sigmoid":
        y = torch.sigmoid(y)
        g = dy * y * (1 - y)
    return {"y": y, "dx": g @ w, "dw": g.T @ x, "db": g.sum(0)}


def _exact_mlp(case, t):
    """The two steps that a pass on a new state makes (one in prepare)."""
    x, y, w = t["x"].double(), t["y"].double(), [v.double() for v in t["w"]]
    b = [torch.zeros(v.shape[0], device=v.device, dtype=v.dtype) for v in w]
    p = w + b
    mom, var = [torch.zeros_like(v) for v in p], [torch.zeros_like(v) for v in p]
    for step in (1, 2):
        h0 = (x @ p[0].T + p[3]).clamp(min=0)
        h1 = torch.sigmoid(h0 @ p[1].T + p[4])
        pred = h1 @ p[2].T + p[5]
        q = torch.softmax(pred, 1)
        loss = -(y * torch.log(q + 1e-8)).sum(1).mean()
        g2 = (q - y) / x.shape[0]
        g1 = (g2 @ p[2]) * h1 * (1 - h1)
        g0 = (g1 @ p[1]) * (h0 > 0)
        grads = [g0.T @ x, g1.T @ h0, g2.T @ h1, g0.sum(0), g1.sum(0), g2.sum(0)]
        for k, g in enumerate(grads):
            mom[k] = 0.9 * mom[k] + 0.1 * g
            var[k] = 0.999 * var[k] + 0.001 * g * g
            p[k] = p[k] - 1e-3 * (mom[k] / (1 - 0.9 ** step)) / ((var[k] / (1 - 0.999 ** step)).sqrt() + 1e-8)
    out = {"pred": pred, "loss": loss}
    for k in range(3):
        out.update({"w%d" % k: p[k], "b%d" % k: p[3 + k], "dw%d" % k: grads[k], "db%d" % k: grads[3 + k]})
    return out


def _exact_grouped(case, t):
    out = {}

    def add(name, v):
        out.setdefault(name, []).append(v.reshape(-1))

    for m in t["models"]:
        x, y, (w0, w1) = m["x"].double(), m["y"].double(), (v.double() for v in m["w"])
        b0, b1 = (torch.zeros(v.shape[0], device=v.device, dtype=v.dtype) for v in (w0, w1))
        for step in (1, 2):
            h = (x @ w0.T + b0).clamp(min=0)
            pred = h @ w1.T + b1
            loss = ((pred - y) ** 2).sum(1).mean()
            g1 = 2 * (pred - y) / x.shape[0]
            g0 = (g1 @ w1) * (h > 0)
            dw0, dw1, db0, db1 = g0.T @ x, g1.T @ h, g0.sum(0), g1.sum(0)
            w0, w1, b0, b1 = w0 - _LR * dw0, w1 - _LR * dw1, b0 - _LR * db0, b1 - _LR * db1
        for name, v in (("pred", pred), ("loss", loss), ("w0", w0), ("b0", b0), ("dw0", dw0), ("db0", db0),
                        ("w2", w1), ("b2", b1), ("dw2", dw1), ("db2", db1)):
            add(name, v)
    return {k: torch.cat(v) for k, v in out.items()}


_EXACT = {"elementwise": _exact_elementwise, "reduce": _exact_reduce, "gather": _exact_gather,
          "matmul": _exact_matmul, "dense": _exact_dense, "mlp": _exact_mlp, "grouped": _exact_grouped}


def _next(s):
    """One xoshiro128++ step of every state (4 int64 rows, 32 bits used):
    the outputs; the states move on in place."""
    m = 0xffffffff
    v = (s[0] + s[3]) & m
    out = ((((v << 7) & m) | (v >> 25)) + s[0]) & m
    t = (s[1] << 9) & m
    s[2] ^= s[0]
    s[3] ^= s[1]
    s[1] ^= s[2]
    s[0] ^= s[3]
    s[2] ^= t
    s[3] = ((s[3] << 11) & m) | (s[3] >> 21)
    return out


def _seeded(size, seed):
    """The generator's documented start states: splitmix64 words for the
    first, and each next one a jump on from the one before.  The jump is
    linear over GF(2), so 2^k of them are one 128 x 128 matrix of bits."""
    m64, words = (1 << 64) - 1, []
    for _ in range(4):
        z = seed = (seed + 0x9e3779b97f4a7c15) & m64
        z = ((z ^ (z >> 30)) * 0xbf58476d1ce4e5b9) & m64
        z = ((z ^ (z >> 27)) * 0x94d049bb133111eb) & m64
        seed = z ^ (z >> 31)
        words.append(seed & 0xffffffff)
    eye = torch.eye(128, dtype=torch.int64, device="cuda").reshape(4, 32, 128)
    bit = torch.arange(32, device="cuda")
    s = (eye << bit[None, :, None]).sum(1)
    acc = torch.zeros_like(s)
    for word in (0x8764000b, 0xf542d2d3, 0x6fa035c3, 0x77f2db5b):
        for b in range(32):
            if word >> b & 1:
                acc ^= s
            _next(s)
        s = acc.clone()
    jump = ((s[:, None, :] >> bit[None, :, None]) & 1).reshape(128, 128).double()
    first = torch.tensor(words, device="cuda")
    states = ((first[:, None] >> bit[None, :]) & 1).reshape(128, 1).double()
    while states.shape[1] < size:
        states = torch.cat([states, (jump @ states) % 2], 1)
        jump = (jump @ jump) % 2
    return (states[:, :size].long().reshape(4, 32, size) << bit[None, :, None]).sum(1)


def _exact_prng(case, seed):
    size, n = case["states"], case["n"]
    if n > 2048 * size:
        return None
    s = _seeded(size, int(seed))

    def stream(count):
        out = []
        for at in range(0, count, size):
            k = min(size, count - at)
            part = s[:, :k].clone()
            out.append(_next(part))
            s[:, :k] = part
        return torch.cat(out)

    u = (stream(n) >> 9).double() / (1 << 23)
    v = (stream(n + n % 2) >> 9).double() / (1 << 23)
    r, a = torch.sqrt(-2 * torch.log(1 - v[0::2])), 2 * math.pi * v[1::2]
    return {"uniform": u, "normal": torch.stack([r * torch.sin(a), r * torch.cos(a)], 1).reshape(-1)[:n],
            "uint32": stream(n).to(torch.int32)}
