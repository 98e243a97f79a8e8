"""What follows a product element by element, written by the launch that writes the product: the same bits as node by node."""
import numpy as np
import pytest

from vkml_b200 import DeviceTensor, DType, NodeDesc, Op, graph
from vkml_b200.backend import Backend

pytestmark = pytest.mark.gpu


def span(b, form, m, k, n):
    rng = np.random.default_rng(m + k + n)
    put = lambda x: DeviceTensor.from_host(b, x)
    x, w = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((k, n), dtype=np.float32)
    x[0, 0] = np.nan
    bias, other = rng.standard_normal(n).astype(np.float32), rng.standard_normal((m, n)).astype(np.float32)
    dx, dw, db, do = put(x.reshape(1, 1, m, k)), put(w.reshape(1, 1, k, n)), put(bias), put(other)
    prod = DeviceTensor.empty(b, (1, 1, m, n))
    y = prod.reshape((m, n))
    new = lambda dtype=DType.F32: DeviceTensor.empty(b, (m, n), dtype)
    nodes, kept = [NodeDesc(int(Op.MATMUL), prod.desc, [dx.desc, dw.desc])], [dx, dw, db, do, prod]
    if form == "where":
        c, z = new(DType.BOOL), new()
        nodes = [NodeDesc(int(Op.LESS_EQUAL), c.desc, [do.desc, db.reshape((1, n)).broadcast_to((m, n)).desc])] + nodes
        nodes.append(NodeDesc(int(Op.WHERE), z.desc, [c.desc, do.desc, y.desc]))
        return nodes, [prod, z], kept + [c]
    add = new()
    nodes.append(NodeDesc(int(Op.ADD), add.desc, [y.desc, db.reshape((1, n)).broadcast_to((m, n)).desc]))
    outs = [prod, add]
    if "mask" in form:
        fa, fb, mask, full = new(), new(), new(DType.BOOL), graph.full_params(0.0)
        nodes += [NodeDesc(int(Op.FULL), fa.desc, [], full), NodeDesc(int(Op.LESS_EQUAL), mask.desc, [add.desc, fa.desc]), NodeDesc(int(Op.FULL), fb.desc, [], full)]
        outs += [fa, mask, fb]
    if "late" in form:
        e = new()
        nodes.append(NodeDesc(int(Op.EXP), e.desc, [do.desc]))
        outs.append(e)
    if "relu" in form:
        r = new()
        nodes.append(NodeDesc(int(Op.RELU), r.desc, [add.desc]))
        outs.append(r)
    return nodes, outs, kept


# one tile and edges of tiles in the small kernel, K in shares; K-slices of the streamed operand and of planes, rows an odd number of words apart
@pytest.mark.parametrize("m,k,n", [(1, 1, 1), (33, 127, 31), (64, 784, 128), (31, 1500, 65), (300, 1900, 101), (93, 1130, 1130), (512, 4096, 260)])
@pytest.mark.parametrize("form", ["where", "add", "add_relu", "add_mask", "add_mask_relu", "add_mask_late_relu"])
def test_epilogue_has_the_nodes_bits(monkeypatch, form, m, k, n):
    results, launches = [], []
    for fuse in ("0", "1"):
        monkeypatch.setenv("VKML_B200_FUSE", fuse)
        b = Backend(0)
        nodes, outs, kept = span(b, form, m, k, n)
        b.set_profiling(True)
        b.compute(nodes)
        launches.append([l for l, _ in b.last_profile()])
        b.set_profiling(False)
        results.append([np.ascontiguousarray(o.numpy()).view(np.uint8) for o in outs])
        del nodes, outs, kept
    for got, want in zip(results[1], results[0]):
        np.testing.assert_array_equal(got, want)
    if form == "where" or (form == "add" and n > 1):  # (a bias of one element is no vector: its add stays a launch)
        assert len(launches[1]) == len(launches[0]) - 1, launches


# a result that lies where the product still reads: the nodes keep their own launches
@pytest.mark.parametrize("m,k", [(33, 33), (70, 130), (128, 1130)])
@pytest.mark.parametrize("side", [0, 1])
def test_results_over_an_operand(monkeypatch, m, k, side):
    results = []
    for fuse in ("0", "1"):
        monkeypatch.setenv("VKML_B200_FUSE", fuse)
        b = Backend(0)
        rng = np.random.default_rng(m + k)
        rows, n = (m, k) if side == 0 else (k, m)  # the result has the shape of the operand that it overwrites
        shapes = [(1, 1, m, k), (1, 1, k, k)] if side == 0 else [(1, 1, k, k), (1, 1, k, m)]
        x, w = (DeviceTensor.from_host(b, rng.standard_normal(s, dtype=np.float32)) for s in shapes)
        prod, bias = DeviceTensor.empty(b, (1, 1, rows, n)), DeviceTensor.from_host(b, rng.standard_normal(n).astype(np.float32))
        over = (x, w)[side].reshape((rows, n))
        b.compute([NodeDesc(int(Op.MATMUL), prod.desc, [x.desc, w.desc]),
                   NodeDesc(int(Op.ADD), over.desc, [prod.reshape((rows, n)).desc, bias.reshape((1, n)).broadcast_to((rows, n)).desc])])
        results.append((prod.numpy(), over.numpy()))
    for got, want in zip(results[1], results[0]):
        np.testing.assert_array_equal(got, want)
