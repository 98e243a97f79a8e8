"""A cross-entropy's nodes, forward and backward, served by the fused passes of loss.cu: every node's value
against the same nodes on their own kernels."""
import numpy as np
import pytest

from vkml_b200 import Backend, DeviceTensor, DType, NodeDesc, Op, graph

pytestmark = pytest.mark.gpu


def loss_nodes(backend, logits, labels, numerator=1.0):
    rows, classes = logits.dims
    nodes, outs = [], []

    def node(op, dims, srcs=(), params=b"", dtype=DType.F32):
        outs.append(DeviceTensor.empty(backend, dims, dtype))
        nodes.append(NodeDesc(int(op), outs[-1].desc, [s.desc for s in srcs], params))
        return outs[-1]

    one, count = node(Op.FULL, (), params=graph.full_params(numerator)), node(Op.FULL, (), params=graph.full_params(rows))
    v = node(Op.DIV, (), [one, count])
    v = node(Op.NEG, (rows,), [node(Op.CONTIGUOUS, (rows,), [v.broadcast_to((rows,))])])
    plane = node(Op.CONTIGUOUS, (rows, classes), [v.reshape((rows, 1)).broadcast_to((rows, classes))])
    wanted = node(Op.CAST, (rows,), [labels])
    index = node(Op.ARANGE, (classes,), params=graph.arange_params(0.0, 1.0))
    hit = node(Op.EQUAL, (rows, classes), [wanted.reshape((rows, 1)).broadcast_to((rows, classes)),
                                           index.broadcast_to((rows, classes))], dtype=DType.BOOL)
    onehot = node(Op.CAST, (rows, classes), [hit])
    picked = node(Op.MUL, (rows, classes), [plane, onehot])
    logp = node(Op.LOG_SOFTMAX, (rows, classes), [logits], graph.axis_params(1))
    prob = node(Op.EXP, (rows, classes), [logp])
    total = node(Op.SUM, (rows, 1), [picked], graph.reduce_params((1,), 2, True))
    node(Op.SUB, (rows, classes), [picked, node(Op.MUL, (rows, classes), [prob, total.broadcast_to((rows, classes))])])
    taken = node(Op.SUM, (rows,), [node(Op.MUL, (rows, classes), [logp, onehot])], graph.reduce_params((1,), 2, False))
    node(Op.MEAN, (), [node(Op.NEG, (rows,), [taken])], graph.reduce_params((0,), 1, False))
    return nodes, outs


def on_both(monkeypatch, x, y, rows, classes, shift, numerator=1.0):
    """Every node's value on the nodes' own kernels and fused."""
    results = {}
    for fuse in ("0", "1"):
        monkeypatch.setenv("VKML_B200_FUSE", fuse)
        b = Backend(0)
        flat = DeviceTensor.from_host(b, x)
        logits = DeviceTensor(b, flat.storage, (rows, classes), (classes * 4, 4), DType.F32, shift * 4)
        nodes, outs = loss_nodes(b, logits, DeviceTensor.from_host(b, y), numerator)
        for o in outs:
            b.copy_from_host(o.storage, 0, np.full(max(o.desc.nbytes, 1), 0x5A, dtype=np.uint8), o.desc.nbytes)
        b.set_profiling(True)
        b.compute(nodes)
        labels = [l for l, _ in b.last_profile()]
        b.set_profiling(False)
        results[fuse] = [o.numpy() for o in outs]
        assert ("fused.loss_value" in labels) == (fuse == "1"), labels
        b.close()
    return results


# one thread, warp and block per row; rows that begin off 16 bytes; register limits and one past them; the
# long-row kernel with rows for some blocks only, and beyond shared memory; one row, one class; a misaligned buffer
@pytest.mark.parametrize("rows,classes,shift", [
    (1, 5, 0), (5, 1, 0), (5000, 10, 0), (129, 32, 0), (9, 33, 0), (300, 257, 0), (100, 1024, 0), (33, 1025, 0), (150, 4095, 0),
    (301, 4097, 0), (20, 51200, 0), (6, 51203, 0), (40, 1000, 1)])
def test_fused_loss(monkeypatch, rows, classes, shift):
    rng = np.random.default_rng(rows * classes)
    x = np.zeros(rows * classes + shift, dtype=np.float32)
    x[shift:] = 4 * rng.standard_normal(rows * classes)
    if rows > 8:
        x[shift + classes:shift + 2 * classes] = -np.inf   # NaN everywhere in that row, as on the CPU
        x[shift + 3 * classes] = np.nan
        x[shift + 4 * classes] = np.inf
    y = rng.integers(0, classes, rows).astype(np.int64)
    results = on_both(monkeypatch, x, y, rows, classes, shift)
    for i, (got, want) in enumerate(zip(results["1"], results["0"])):
        np.testing.assert_allclose(got, want, rtol=2e-5, atol=2e-6 / rows, err_msg=str(i))


# a scale that is not finite makes every element off the label a NaN, and with it the row's sum; a label that is no class picks nothing
@pytest.mark.parametrize("numerator", [1.0, np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("rows,classes,shift", [(5, 1, 0), (200, 10, 0), (40, 257, 0), (20, 3000, 0), (5, 5000, 0), (20, 70, 1)])
def test_scales_and_labels_outside_the_usual(monkeypatch, rows, classes, shift, numerator):
    rng = np.random.default_rng(rows + classes)
    x = rng.standard_normal(rows * classes + shift).astype(np.float32)
    y = rng.integers(0, classes, rows).astype(np.int64)
    y[1], y[2], y[3] = classes, -1, 1 << 40
    results = on_both(monkeypatch, x, y, rows, classes, shift, numerator)
    for i, (got, want) in enumerate(zip(results["1"], results["0"])):
        np.testing.assert_allclose(got, want, rtol=2e-5, atol=2e-6 / rows, err_msg=str(i))
