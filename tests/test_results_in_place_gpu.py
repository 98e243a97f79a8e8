"""What follows a product may lie over the product's result: the launch that serves both writes the later value last."""
import numpy as np
import pytest

from vkml_b200 import DeviceTensor, DType, NodeDesc, Op, graph

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def backend():
    import vkml_b200
    b = vkml_b200.Backend(0)
    yield b
    b.close()


def layer(b, x, w, bias, dtype, form, place):
    """The nodes' last result, in a buffer of its own or over the one that `place` names."""
    (m, k), n = x.shape, w.shape[1]
    dx, dw, db = DeviceTensor.from_host(b, x.reshape(1, 1, m, k)), DeviceTensor.from_host(b, w.reshape(1, 1, k, n)), DeviceTensor.from_host(b, bias)
    y, z, last = (DeviceTensor.empty(b, (m, n), dtype) for _ in range(3))
    wide = db.reshape((1, n)).broadcast_to((m, n))
    last = {"own": last, "product": y, "sum": z}[place]
    nodes = [NodeDesc(int(Op.MATMUL), y.reshape((1, 1, m, n)).desc, [dx.desc, dw.desc])]
    if form == "add":
        nodes.append(NodeDesc(int(Op.ADD), last.desc, [y.desc, wide.desc]))
    elif form == "relu":
        nodes += [NodeDesc(int(Op.ADD), z.desc, [y.desc, wide.desc]), NodeDesc(int(Op.RELU), last.desc, [z.desc])]
    else:
        other = np.random.default_rng(m).standard_normal((m, n)).astype(np.float32)
        do, c = DeviceTensor.from_host(b, other), DeviceTensor.empty(b, (m, n), DType.BOOL)
        nodes = [NodeDesc(int(Op.LESS_EQUAL), c.desc, [do.desc, wide.desc])] + nodes
        nodes.append(NodeDesc(int(Op.WHERE), last.desc, [c.desc, do.desc, y.desc]))
    b.compute(nodes)
    return last.numpy()


FORMS = [("add", "product"), ("relu", "product"), ("relu", "sum"), ("where", "product")]


# the small kernel, one share of K and several; the streamed operand's and the planes' fold
@pytest.mark.parametrize("m,k,n", [(33, 127, 31), (31, 1500, 65), (64, 784, 128), (300, 1900, 101), (93, 1130, 1130), (512, 4096, 260)])
@pytest.mark.parametrize("form,place", FORMS)
def test_fp32(backend, m, k, n, form, place):
    rng = np.random.default_rng(m + n)
    x, w, bias = (rng.standard_normal(s, dtype=np.float32) for s in ((m, k), (k, n), (n,)))
    own = layer(backend, x, w, bias, DType.F32, form, "own")
    got = layer(backend, x, w, bias, DType.F32, form, place)
    assert np.array_equal(got.view(np.uint32), own.view(np.uint32))


# rows that TMA does not read, without and with slices of K; rows that it reads
@pytest.mark.parametrize("m,k,n", [(247, 348, 1369), (40, 4099, 300), (512, 512, 640), (64, 4096, 1024)])
@pytest.mark.parametrize("form,place", FORMS[:3])
def test_half(backend, m, k, n, form, place):
    rng = np.random.default_rng(m + n)
    x, w, bias = (rng.standard_normal(s).astype(np.float16) for s in ((m, k), (k, n), (n,)))
    own = layer(backend, x, w, bias, DType.F16, form, "own")
    got = layer(backend, x, w, bias, DType.F16, form, place)
    assert np.array_equal(got.view(np.uint16), own.view(np.uint16))


# what a where chooses from, filled with one value in the span and read as one word, or filled before it and read whole
@pytest.mark.parametrize("m,k,n", [(33, 127, 31), (64, 784, 128), (300, 1900, 101), (512, 4096, 260)])
def test_a_filled_choice(backend, m, k, n):
    rng = np.random.default_rng(m)
    x, w, c = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((k, n), dtype=np.float32), rng.random((m, n)) < 0.5
    dx, dw, dc = DeviceTensor.from_host(backend, x.reshape(1, 1, m, k)), DeviceTensor.from_host(backend, w.reshape(1, 1, k, n)), DeviceTensor.from_host(backend, c)
    y = DeviceTensor.empty(backend, (1, 1, m, n))
    results = []
    for inside in (True, False):
        f, z = DeviceTensor.empty(backend, (m, n)), DeviceTensor.empty(backend, (m, n))
        fill = NodeDesc(int(Op.FULL), f.desc, [], graph.full_params(-0.5))
        nodes = [NodeDesc(int(Op.MATMUL), y.desc, [dx.desc, dw.desc]), NodeDesc(int(Op.WHERE), z.desc, [dc.desc, f.desc, y.reshape((m, n)).desc])]
        if inside:
            backend.compute([fill] + nodes)
        else:
            backend.compute([fill])
            backend.compute(nodes)
        results.append(z.numpy())
        assert np.array_equal(results[-1], np.where(c, np.float32(-0.5), y.numpy().reshape(m, n)))
    assert np.array_equal(*results)


# a product of the wrong rank is refused, with something behind it as without
@pytest.mark.parametrize("dims", [(), (8,), (2, 4), (1, 2, 4)])
@pytest.mark.parametrize("behind", [False, True])
def test_a_product_of_another_rank_is_refused(backend, dims, behind):
    from vkml_b200.backend import ShapeError
    a, b, y = (DeviceTensor.empty(backend, dims) for _ in range(3))
    nodes = [NodeDesc(int(Op.MATMUL), y.desc, [a.desc, b.desc])]
    if behind:
        nodes.append(NodeDesc(int(Op.ADD), DeviceTensor.empty(backend, dims).desc, [y.desc, a.desc]))
    with pytest.raises(ShapeError):
        backend.compute(nodes)
