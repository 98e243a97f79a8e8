"""The work that programs on this backend are made of, as timed cases.

Every case is a program of graph nodes built the way vkML's graph and autograd layers emit them and
handed to the public entry points of `vkml_b200.Backend`:

  matmul         one product through `Backend.compute`: the squares, the skinny and the long-K product of
                 the GEMM sweep in `bench.py`, and sizes that are no multiple of anything
  linear_f16     a Linear layer (product, bias, ReLU) over F16 storage
  cross_entropy  the loss of a classifier, forward and backward, at the (rows, classes) of the configurations
  embedding      rows of a table selected by an index list, and the table's gradient
  mlp, cnn       whole training steps: forward, loss, backward, SGD with momentum, parameters assigned

A node leaves its value in a buffer of its own, so the bytes that a program cannot do without are its
inputs read once and every node's result written once.
"""
import math
import types

import torch

from vkml_b200 import Backend, DeviceTensor, DType, NodeDesc, Op, graph

_TORCH = {DType.F32: ("<f4", torch.float32), DType.F16: ("<f2", torch.float16), DType.I64: ("<i8", torch.int64),
          DType.I32: ("<i4", torch.int32), DType.BOOL: ("|u1", torch.uint8)}


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _matmul(name, m, k, n, layout="nn", batch=1):
    return {"name": name, "kind": "matmul", "m": m, "k": k, "n": n, "layout": layout, "batch": batch}


def listed():
    return [
        # the smallest square of the sweep: one call, its latency
        _matmul("matmul 256", 256, 256, 256),
        # a Linear layer's product, x . W^T, with sizes that divide into no tile and pitches that are not 16 bytes
        _matmul("matmul ragged", 1000, 1433, 777, "nt"),
        # a few rows through a large weight (inference on a small batch)
        _matmul("matmul skinny", 64, 4096, 4096),
        # a small result from a long reduction (a weight gradient over many samples)
        _matmul("matmul long k", 512, 65536, 512),
        # the headline of the sweep: bound by the tensor cores
        _matmul("matmul 8192", 8192, 8192, 8192),
        # half storage, as a model kept in F16 runs its hidden layers
        {"name": "linear f16", "kind": "linear_f16", "m": 2048, "k": 4096, "n": 4096},
        # the losses of the configurations: many rows of few classes, and a vocabulary
        {"name": "cross entropy 65536x10", "kind": "cross_entropy", "rows": 65536, "classes": 10},
        {"name": "cross entropy 1024x32000", "kind": "cross_entropy", "rows": 1024, "classes": 32000},
        # an Embedding, forward and backward, as the memory-bound table of the benchmark sizes it
        {"name": "embedding 50000x1024", "kind": "embedding", "vocab": 50000, "width": 1024, "count": 8192},
        # the training steps of the configurations
        {"name": "mlp 784-128-10 b64", "kind": "mlp", "batch": 64, "inputs": 784, "hidden": 128, "layers": 2,
         "classes": 10},
        {"name": "mlp 4096-8192x3-1000 b2048", "kind": "mlp", "batch": 2048, "inputs": 4096, "hidden": 8192,
         "layers": 4, "classes": 1000},
        {"name": "cnn 32x32 b256", "kind": "cnn", "batch": 256, "cin": 3, "hw": 32, "c1": 64, "c2": 128, "c3": 256,
         "classes": 100},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One case of the ranges between the listed ones: sizes over their logarithm, mostly odd ones."""
    kind = rng.choice(["matmul"] * 4 + ["linear_f16", "cross_entropy", "cross_entropy", "embedding", "mlp", "mlp", "cnn"])
    if kind == "matmul":
        while True:
            batch = rng.choice([1, 1, 1, _log(rng, 2, 64)])
            m, n, k = _log(rng, 64, 8192), _log(rng, 64, 8192), _log(rng, 64, 65536)
            if rng.random() < 0.4:  # as often as not a model's sizes are multiples of something
                m, n, k = (64 * max(1, v // 64) for v in (m, n, k))
            if 256 ** 3 <= batch * m * n * k <= 2e11 and batch * (m * k + k * n + m * n) <= 3e8:
                return {"kind": kind, "m": m, "k": k, "n": n, "layout": rng.choice(["nn", "nt", "tn"]), "batch": batch}
    if kind == "linear_f16":
        return {"kind": kind, "m": _log(rng, 64, 4096), "k": _log(rng, 256, 8192), "n": _log(rng, 256, 8192)}
    if kind == "cross_entropy":
        classes = _log(rng, 10, 32000)
        return {"kind": kind, "rows": _log(rng, 256, min(65536, 3.3e7 / classes)), "classes": classes}
    if kind == "embedding":
        return {"kind": kind, "vocab": _log(rng, 2000, 60000), "width": _log(rng, 32, 1024), "count": _log(rng, 512, 16384)}
    if kind == "mlp":
        return {"kind": kind, "batch": _log(rng, 32, 2048), "inputs": _log(rng, 64, 4096), "hidden": _log(rng, 64, 4096),
                "layers": rng.choice([2, 3, 4]), "classes": _log(rng, 10, 1000)}
    c1 = rng.choice([16, 24, 32, 48, 64])
    return {"kind": "cnn", "batch": _log(rng, 16, 256), "cin": rng.choice([1, 3, 4]), "hw": rng.choice([24, 28, 30, 32]),
            "c1": c1, "c2": 2 * c1, "c3": rng.choice([2, 4]) * c1, "classes": _log(rng, 10, 200)}


# ---------------------------------------------------------------------------
# a program: spans of nodes over buffers of the backend, and device copies between them
# ---------------------------------------------------------------------------

class _Paper:
    """Stands in for the backend where a program is only counted: hands out addresses, no memory."""

    def __init__(self):
        self.at = 1 << 20

    def allocate(self, nbytes):
        self.at += (nbytes + 511) // 512 * 512 + 512
        return types.SimpleNamespace(data=self.at, nbytes=nbytes)


_backend = None


def _gpu():
    global _backend
    if _backend is None:
        _backend = Backend(0)
    return _backend


def _tensor(t):
    """A dense device tensor of the backend as the torch tensor over the same memory."""
    kind, dtype = _TORCH[t.dtype]
    if t.numel == 0:
        return torch.empty(t.dims, dtype=dtype, device="cuda")
    face = types.SimpleNamespace(keep=t, __cuda_array_interface__={
        "shape": t.dims, "typestr": kind, "data": (t.desc.data, False), "strides": None, "version": 3})
    return torch.as_tensor(face, device="cuda")


def _mat(t, batch=None):
    """Matmul operands are rank 4: a matrix, broadcast over `batch` where one is given."""
    if len(t.dims) == 2:
        t = DeviceTensor(t.backend, t.storage, (1, 1) + t.dims, (0, 0) + t.strides, t.dtype, t.offset)
    elif len(t.dims) == 3:
        t = DeviceTensor(t.backend, t.storage, (1,) + t.dims, (0,) + t.strides, t.dtype, t.offset)
    return t if batch is None else t.broadcast_to((1, batch) + t.dims[2:])


class Program:
    def __init__(self, backend):
        self.backend = backend
        self.parts = []      # ("compute", nodes) and ("copy", [(to, from)])
        self.odd = {}        # parts whose nodes differ in every second pass: index -> nodes
        self.inputs = []     # (tensor, how its values are drawn)
        self.results = []    # of every node
        self.copied = []
        self.flops = 0.0
        self.unread = 0      # bytes of the inputs that the program does not read
        self.outputs = {}

    def input(self, dims, how, dtype=DType.F32):
        t = DeviceTensor.empty(self.backend, dims, dtype)
        self.inputs.append((t, how))
        return t

    def span(self):
        self.parts.append(("compute", []))

    def copy(self, pairs):
        self.parts.append(("copy", pairs))
        self.copied += [to for to, _ in pairs]

    def node(self, op, dims, srcs=(), params=b"", dtype=DType.F32):
        out = DeviceTensor.empty(self.backend, dims, dtype)
        self.node_into(op, out, srcs, params)
        return out

    def node_into(self, op, out, srcs, params=b""):
        self.parts[-1][1].append(NodeDesc(int(op), out.desc, [s.desc for s in srcs], params))
        self.results.append(out)
        self.flops += out.numel

    def matmul(self, a, b, batch=None):
        """a[.., m, k] . b[.., k, n]; rank-2 operands give a rank-2 result."""
        ra, rb = _mat(a, batch), _mat(b, batch if len(b.dims) == 2 else None)
        dims = ra.dims[:3] + rb.dims[3:]
        out = self.node(Op.MATMUL, dims, [ra, rb], dtype=a.dtype)
        self.flops += 2.0 * out.numel * ra.dims[3]
        return out.reshape(dims[2:] if batch is None and dims[0] * dims[1] == 1 else dims[1:])

    def full(self, dims, value):
        return self.node(Op.FULL, dims, params=graph.full_params(value))

    def sum(self, t, axes, keepdim=True):
        dims = tuple(1 if i in axes else d for i, d in enumerate(t.dims) if keepdim or i not in axes)
        return self.node(Op.SUM, dims, [t], graph.reduce_params(axes, len(t.dims), keepdim))

    # -- pieces that every model is made of --
    def loss_head(self, labels, rows, classes):
        """The one-hot rows scaled by -1/rows that the loss is differentiated with."""
        one, count = self.full((), 1.0), self.full((), float(rows))
        scale = self.node(Op.DIV, (), [one, count])
        scale = self.node(Op.CONTIGUOUS, (rows,), [scale.broadcast_to((rows,))])
        scale = self.node(Op.NEG, (rows,), [scale])
        scale = self.node(Op.CONTIGUOUS, (rows, classes), [scale.reshape((rows, 1)).broadcast_to((rows, classes))])
        wanted = self.node(Op.CAST, (rows,), [labels])
        index = self.node(Op.ARANGE, (classes,), params=graph.arange_params(0.0, 1.0))
        hit = self.node(Op.EQUAL, (rows, classes), [wanted.reshape((rows, 1)).broadcast_to((rows, classes)),
                                                    index.broadcast_to((rows, classes))], dtype=DType.BOOL)
        onehot = self.node(Op.CAST, (rows, classes), [hit])
        return onehot, self.node(Op.MUL, (rows, classes), [scale, onehot])

    def loss_backward(self, logits, picked):
        dims = logits.dims
        logp = self.node(Op.LOG_SOFTMAX, dims, [logits], graph.axis_params(1))
        prob = self.node(Op.EXP, dims, [logp])
        total = self.sum(picked, (1,))
        share = self.node(Op.MUL, dims, [prob, total.broadcast_to(dims)])
        return logp, self.node(Op.SUB, dims, [picked, share])

    def loss_value(self, logp, onehot):
        rows = logp.dims[0]
        taken = self.node(Op.MUL, logp.dims, [logp, onehot])
        taken = self.sum(taken, (1,), keepdim=False)
        taken = self.node(Op.NEG, (rows,), [taken])
        return self.node(Op.MEAN, (), [taken], graph.reduce_params((0,), 1, False))

    def relu_mask(self, t):
        mask = self.node(Op.LESS_EQUAL, t.dims, [t, self.full(t.dims, 0.0)], dtype=DType.BOOL)
        return mask, self.full(t.dims, 0.0)

    def work(self):
        read = sum(t.desc.nbytes for t, _ in self.inputs) - self.unread
        kept = sum(c.desc.nbytes for c in self.copied)
        return {"bytes": float(read + kept + sum(r.desc.nbytes for r in self.results)), "flops": self.flops}

    def sgd(self, params, grads, lr):
        """v = 0.9 v + g, then p = p - lr v, then the new parameters assigned.  The velocities change
        places from pass to pass, as a new result does with the one it replaces."""
        first = [self.input(p.dims, ("uniform", -1e-3, 1e-3)) for p in params]
        second = [DeviceTensor.empty(self.backend, p.dims) for p in params]
        stepped = [DeviceTensor.empty(self.backend, p.dims) for p in params]
        self.span()
        for v, w, g in zip(second, first, grads):
            self.node_into(Op.SCALED_ADD, v, [w, g], graph.scaled_add_params(0.9, 1.0))
        self.odd[len(self.parts) - 1] = [
            NodeDesc(int(Op.SCALED_ADD), v.desc, [w.desc, g.desc], graph.scaled_add_params(0.9, 1.0))
            for v, w, g in zip(first, second, grads)]
        self.span()
        for q, p, v in zip(stepped, params, second):
            self.node_into(Op.SCALED_ADD, q, [p, v], graph.scaled_add_params(1.0, -lr))
        self.odd[len(self.parts) - 1] = [
            NodeDesc(int(Op.SCALED_ADD), q.desc, [p.desc, v.desc], graph.scaled_add_params(1.0, -lr))
            for q, p, v in zip(stepped, params, first)]
        self.copy(list(zip(params, stepped)))
        return first, second


# ---------------------------------------------------------------------------
# the programs of the cases
# ---------------------------------------------------------------------------

def _build_matmul(p, c):
    m, k, n, layout = c["m"], c["k"], c["n"], c["layout"]
    lead = (c["batch"],) if c["batch"] > 1 else ()
    a = p.input(lead + ((k, m) if layout == "tn" else (m, k)), ("normal", 1.0))
    b = p.input(lead + ((n, k) if layout == "nt" else (k, n)), ("normal", 1.0))
    p.span()
    r = len(lead)
    p.outputs["c"] = p.matmul(a.transpose(r, r + 1) if layout == "tn" else a, b.transpose(r, r + 1) if layout == "nt" else b,
                              c["batch"] if lead else None)


def _build_linear_f16(p, c):
    m, k, n = c["m"], c["k"], c["n"]
    x = p.input((m, k), ("normal", 1.0), DType.F16)
    w = p.input((n, k), ("uniform", -1 / math.sqrt(k), 1 / math.sqrt(k)), DType.F16)
    bias = p.input((n,), ("uniform", -1 / math.sqrt(k), 1 / math.sqrt(k)), DType.F16)
    p.span()
    y = p.matmul(x, w.transpose(0, 1))
    z = p.node(Op.ADD, (m, n), [y, bias.broadcast_to((m, n))], dtype=DType.F16)
    p.outputs = {"y": y, "z": z, "h": p.node(Op.RELU, (m, n), [z], dtype=DType.F16)}


def _build_cross_entropy(p, c):
    rows, classes = c["rows"], c["classes"]
    logits = p.input((rows, classes), ("normal", 2.0))
    labels = p.input((rows,), ("index", classes), DType.I64)
    p.span()
    onehot, picked = p.loss_head(labels, rows, classes)
    logp, grad = p.loss_backward(logits, picked)
    p.span()
    p.outputs = {"loss": p.loss_value(logp, onehot), "log_probabilities": logp, "gradient": grad, "onehot": onehot,
                 "picked": picked}


def _build_embedding(p, c):
    vocab, width, count = c["vocab"], c["width"], c["count"]
    table = p.input((vocab, width), ("normal", 1.0))
    index = p.input((count,), ("index", vocab), DType.I64)
    grad = p.input((count, width), ("normal", 1e-2))
    p.unread = max(0, vocab - count) * width * 4
    p.span()
    p.outputs["rows"] = p.node(Op.INDEX_SELECT, (count, width), [table, index], graph.axis_params(0))
    p.span()
    p.outputs["table_gradient"] = p.node(Op.SCATTER_ADD, (vocab, width), [grad, index], graph.axis_params(0))


def _weights(p, out, inner, dims=None):
    bound = 1 / math.sqrt(inner)
    return p.input(dims or (out, inner), ("uniform", -bound, bound)), p.input((out,), ("uniform", -bound, bound))


def _finish(p, params, grads, logp, onehot):
    """The rest of a training step behind its backward pass: optimiser, assignment, loss."""
    grads = [g.reshape(w.dims) if g.is_contiguous() else g for g, w in zip(grads, params)]
    first, second = p.sgd(params, grads, 0.01)
    p.span()
    p.outputs["loss"] = p.loss_value(logp, onehot)
    for name, group in (("parameter", params), ("gradient", grads), ("velocity", second), ("velocity_before", first)):
        for i, t in enumerate(group):
            p.outputs["%s_%02d" % (name, i)] = t


def _build_mlp(p, c):
    batch = c["batch"]
    widths = [c["inputs"]] + [c["hidden"]] * (c["layers"] - 1) + [c["classes"]]
    x = p.input((batch, widths[0]), ("uniform", 0.0, 1.0) if c["hidden"] < 1024 else ("normal", 1.0))
    labels = p.input((batch,), ("index", c["classes"]), DType.I64)
    layers = [_weights(p, o, i) for i, o in zip(widths[:-1], widths[1:])]
    p.span()
    acts, masks = [x], []
    for i, (w, b) in enumerate(layers):
        y = p.matmul(acts[-1], w.transpose(0, 1))
        y = p.node(Op.ADD, y.dims, [y, b.broadcast_to(y.dims)])
        if i + 1 < len(layers):
            masks.append(p.relu_mask(y))
            if i + 2 == len(layers):
                onehot, picked = p.loss_head(labels, batch, c["classes"])
            acts.append(p.node(Op.RELU, y.dims, [y]))
    logp, g = p.loss_backward(y, picked)
    grads_out = [g]
    for (w, _), (mask, zeros) in zip(reversed(layers[1:]), reversed(masks)):
        g = p.matmul(g, w)
        g = p.node(Op.WHERE, g.dims, [mask, zeros, g])
        grads_out.insert(0, g)
    grads = []
    for a, g in zip(acts, grads_out):
        grads += [p.matmul(a.transpose(0, 1), g).transpose(0, 1), p.sum(g, (0,))]
    _finish(p, [t for pair in layers for t in pair], grads, logp, onehot)


def _build_cnn(p, c):
    batch, hw, classes = c["batch"], c["hw"], c["classes"]
    widths, convs = [c["cin"], c["c1"], c["c2"], c["c3"]], []
    x = p.input((batch, c["cin"], hw, hw), ("uniform", 0.0, 1.0))
    labels = p.input((batch,), ("index", classes), DType.I64)
    weights = [_weights(p, o, 9 * i) for i, o in zip(widths[:-1], widths[1:])]
    flat = widths[3] * (hw // 8) ** 2
    weights.append(_weights(p, classes, flat))
    p.span()
    h = x
    for i in range(3):
        w, b = weights[i]
        cout, side = widths[i + 1], h.dims[2]
        unfold = graph.unfold_params((3, 3), (1, 1), (1, 1), (1, 1), (side, side))
        pool = graph.unfold_params((2, 2), (2, 2), (0, 0), (1, 1), (side, side))
        cols = p.node(Op.IM2COL, (batch, 9 * widths[i], side * side), [h], unfold)
        y = p.matmul(w, cols, batch).reshape((batch, cout, side, side))
        y = p.node(Op.ADD, y.dims, [y, b.reshape((cout, 1, 1)).broadcast_to(y.dims)])
        if i == 2:
            mask = p.relu_mask(y)
            onehot, picked = p.loss_head(labels, batch, classes)
        r = p.node(Op.RELU, y.dims, [y])
        h = p.node(Op.MAX_POOL2D, (batch, cout, side // 2, side // 2), [r], pool)
        convs.append((cols, y, r, h, unfold, pool))
    feats = h.reshape((batch, flat))
    head, head_bias = weights[3]
    y = p.matmul(feats, head.transpose(0, 1))
    y = p.node(Op.ADD, y.dims, [y, head_bias.broadcast_to(y.dims)])
    logp, g_head = p.loss_backward(y, picked)
    g = p.matmul(g_head, head).reshape(h.dims)
    grads, bias_in = [None] * 4, [None] * 3
    for i in (2, 1, 0):
        cols, y, r, h, unfold, pool = convs[i]
        if i < 2:
            mask = p.relu_mask(y)
            wide = p.matmul(weights[i + 1][0].transpose(0, 1), g_conv, batch)
            g = p.node(Op.COL2IM, h.dims, [wide], convs[i + 1][4])
        g = p.node(Op.MAX_POOL2D_BACKWARD, r.dims, [g, r], pool)
        g = p.node(Op.WHERE, r.dims, [mask[0], mask[1], g])
        bias_in[i] = g
        g_conv = g.reshape((batch, r.dims[1], r.dims[2] * r.dims[3]))
        each = p.matmul(g_conv, cols.transpose(1, 2), batch)
        grads[i] = p.sum(each.reshape((1,) + each.dims), (1,))
    biases = [p.sum(t, (0, 2, 3)) for t in bias_in]
    grads[3] = p.matmul(feats.transpose(0, 1), g_head).transpose(0, 1)
    biases.append(p.sum(g_head, (0,)))
    _finish(p, [t for pair in weights for t in pair], [t for pair in zip(grads, biases) for t in pair], logp, onehot)


_BUILD = {"matmul": _build_matmul, "linear_f16": _build_linear_f16, "cross_entropy": _build_cross_entropy,
          "embedding": _build_embedding, "mlp": _build_mlp, "cnn": _build_cnn}


def _program(case, backend):
    p = Program(backend)
    _BUILD[case["kind"]](p, case)
    return p


# ---------------------------------------------------------------------------
# what is timed
# ---------------------------------------------------------------------------

def prepare(case, seed):
    """The inputs in device memory and, for the programs that a user runs many times, their spans packed once."""
    backend = _gpu()
    backend.synchronize()  # buffers of an earlier state may be handed out again below
    p = _program(case, backend)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    for t, how in p.inputs:
        view = _tensor(t)
        if how[0] == "index":
            view.copy_(torch.randint(0, how[1], t.dims, generator=gen, device="cuda"))
        elif how[0] == "normal":
            view.copy_(torch.randn(t.dims, generator=gen, device="cuda") * how[1])
        else:
            view.copy_(torch.rand(t.dims, generator=gen, device="cuda") * (how[2] - how[1]) + how[1])
    packed = case["kind"] in ("cross_entropy", "mlp", "cnn")
    passes = []
    for odd in (False, True) if p.odd else (False,):
        calls = []
        for i, (what, part) in enumerate(p.parts):
            if what == "copy":
                calls.append(("copy", [(d.storage, 0, s.storage, 0, d.desc.nbytes) for d, s in part]))
            else:
                nodes = p.odd.get(i, part) if odd else part
                calls.append(("packed", graph.pack_nodes(nodes), len(nodes)) if packed else ("nodes", nodes))
        passes.append(calls)
    # (where an output is a view, the matrix that it is the transpose of)
    outputs = {name: _tensor(t if t.is_contiguous() else t.transpose(0, 1)) for name, t in p.outputs.items()}
    torch.cuda.synchronize()
    return {"backend": backend, "program": p, "passes": passes, "at": 0, "outputs": outputs}


def run(state):
    backend = state["backend"]
    calls = state["passes"][state["at"] % len(state["passes"])]
    state["at"] += 1
    for call in calls:
        if call[0] == "packed":
            backend.compute_packed(call[1], call[2])
        elif call[0] == "nodes":
            backend.compute(call[1])
        else:
            backend.copy_device_to_device(call[1])
    return state["outputs"]


def work(case):
    return _program(case, _Paper()).work()


def tolerance(case):
    kind = case["kind"]
    if kind == "embedding":
        return "exact"  # rows are moved, and those of one destination added in the order of the indices
    if kind == "matmul":
        # the tensor core's fp32 accumulator truncates: an error that grows with the length of its chain of
        # additions, 4e-6 at K = 1024 and 6e-5 at K = 8192 and above
        return {"rel": min(1e-4, max(1e-5, 1e-4 * case["k"] / 8192)), "max": 1e-3}
    if kind == "linear_f16":
        # one result in a hundred or so rounds to the neighbouring half (2^-10 of the value), and y + bias rounds again
        return {"rel": 5e-4, "max": 4e-3}
    if kind == "cross_entropy":
        return {"rel": 1e-5, "max": 1e-4}
    # A ReLU or a pooling maximum decided by the last bits of a product switches one path of the gradient on or
    # off: a share s of switched units moves the gradient by about sqrt(s).  (Measured between the tensor cores
    # and plain fp32 arithmetic, after two passes: 7e-3 and 0.4 for the wide MLP, 2e-3 and 0.07 for the CNN.)
    return {"rel": 1e-2, "max": 0.5}
