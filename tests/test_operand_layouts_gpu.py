"""Products whose kernels read the caller's operands themselves, over operands that are not one dense matrix."""
import os

import numpy as np
import pytest

from vkml_b200 import DeviceTensor, DType, NodeDesc, Op

pytestmark = pytest.mark.gpu


def context(value):
    import vkml_b200
    os.environ["VKML_B200_GEMM_INLINE"] = value
    b = vkml_b200.Backend(0)
    del os.environ["VKML_B200_GEMM_INLINE"]
    return b


# the largest pitch that TF32 terms are split at inside the kernel, and the first that planes serve; rows 32 and 64 of the right operand's tile are used
@pytest.mark.parametrize("pitch", [(1 << 24) - 4, 1 << 24])
def test_rows_far_apart(pitch):
    b = context("8")  # (TF32 terms inside the kernel wherever they fit)
    m, k, n = 300, 1024, 72
    rng = np.random.default_rng(pitch)
    x, w = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((n, k), dtype=np.float32)
    dx, wide = DeviceTensor.from_host(b, x.reshape(1, 1, m, k)), DeviceTensor.empty(b, (n, pitch))
    for row in range(n):
        b.copy_from_host(wide.storage, 4 * row * pitch, w[row])
    dw = DeviceTensor(b, wide.storage, (1, 1, k, n), (0, 0, 4, 4 * pitch), wide.dtype, 0)
    out = DeviceTensor.empty(b, (1, 1, m, n))
    b.compute([NodeDesc(int(Op.MATMUL), out.desc, [dx.desc, dw.desc])])
    want, terms = x.astype(np.float64) @ w.T.astype(np.float64), np.abs(x).astype(np.float64) @ np.abs(w.T).astype(np.float64)
    assert np.all(np.abs(out.numpy().reshape(m, n) - want) <= (k / 8 / 4 * 2.0 ** -23 + 2.0 ** -20) * terms)
    b.close()


@pytest.fixture(scope="module")
def backend():
    b = context("auto")
    yield b
    b.close()


def half_layer(b, x, w, bias, over, relu):
    """A Linear layer over half storage; `over`: what the last result (the sum, or relu's) lies over."""
    (m, k), n = x.shape, w.shape[1]
    dx, dw, db = DeviceTensor.from_host(b, x.reshape(1, 1, m, k)), DeviceTensor.from_host(b, w.reshape(1, 1, k, n)), DeviceTensor.from_host(b, bias)
    y, z, h = (DeviceTensor.empty(b, (m, n), DType.F16) for _ in range(3))
    place = {None: None, "x": dx, "w": dw, "product": y, "sum": z}[over]
    if place is not None and relu:
        h = place.reshape((m, n))
    elif place is not None:
        z = place.reshape((m, n))
    nodes = [NodeDesc(int(Op.MATMUL), y.reshape((1, 1, m, n)).desc, [dx.desc, dw.desc]),
             NodeDesc(int(Op.ADD), z.desc, [y.desc, db.reshape((1, n)).broadcast_to((m, n)).desc])]
    if relu:
        nodes.append(NodeDesc(int(Op.RELU), h.desc, [z.desc]))
    b.compute(nodes)
    return (h if relu else z).numpy()


# rows that TMA reads and rows that it does not, one slice of K and several; over an operand the nodes keep their own launches, over a result of the
# layer they are still one
@pytest.mark.parametrize("side", [301, 517, 640, 131])
@pytest.mark.parametrize("over,relu", [("x", True), ("x", False), ("w", True), ("w", False), ("product", True), ("product", False), ("sum", True)])
def test_half_layers_over_their_operands(backend, side, over, relu):
    rng = np.random.default_rng(side)
    m = k = n = side  # (the result has the shape of either operand)
    if side == 131:
        m, k, n = (40, 1500, 1500) if over != "w" else (1500, 1500, 40)
    x, w = (rng.standard_normal(s).astype(np.float16) for s in ((m, k), (k, n)))
    bias = rng.standard_normal(n).astype(np.float16)
    want = half_layer(backend, x, w, bias, None, relu)
    for _ in range(3):
        got = half_layer(backend, x, w, bias, over, relu)
        assert np.array_equal(got.view(np.uint16), want.view(np.uint16))


# the small kernel; TF32 and half terms split inside the kernel, half terms from planes, the streamed operand; halves that TMA reads and does not
@pytest.mark.parametrize("dtype,m,k", [("f4", 33, 33), ("f4", 97, 130), ("f4", 512, 512), ("f4", 301, 1003), ("f4", 1400, 1204), ("f4", 4096, 768), ("f4", 64, 4096),
                                       ("f2", 301, 301), ("f2", 768, 512), ("f2", 40, 1500), ("f2", 2050, 517)])
@pytest.mark.parametrize("side", [0, 1])
@pytest.mark.parametrize("turned", [False, True])
def test_products_over_their_operand(backend, dtype, m, k, side, turned):
    rng = np.random.default_rng(m + k)
    shapes = [(m, k), (k, k)] if side == 0 else [(k, k), (k, m)]
    a, b = (rng.standard_normal(s).astype(dtype) for s in shapes)
    results = []
    for over in (False, True, True):
        put = [DeviceTensor.from_host(backend, t.reshape((1, 1) + t.shape)) for t in (a, b)]
        if turned:  # the operand that is not written over, stored the other way round
            t = (a, b)[1 - side]
            put[1 - side] = DeviceTensor.from_host(backend, np.ascontiguousarray(t.T).reshape((1, 1) + t.T.shape)).transpose(2, 3)
        out = put[side] if over else DeviceTensor.empty(backend, (1, 1, a.shape[0], b.shape[1]), put[0].dtype)
        backend.compute([NodeDesc(int(Op.MATMUL), out.desc, [t.desc for t in put])])
        results.append(out.numpy().astype(np.float64))
    want, terms = a.astype(np.float64) @ b.astype(np.float64), np.abs(a).astype(np.float64) @ np.abs(b).astype(np.float64)
    rounding = 2.0 ** -11 * np.abs(want) if dtype == "f2" else 0  # (widened copies add in another order: neighbours may differ)
    for got in results:
        assert np.all(np.abs(got.reshape(want.shape) - want) <= (k / 8 / 4 * 2.0 ** -23 + 2.0 ** -20) * terms + rounding)
    if dtype == "f4":
        assert np.array_equal(results[0], results[1]) and np.array_equal(results[0], results[2])


def test_a_span_reads_what_was_written_over_an_operand(backend):
    """x . w, x <- x . w, x . w again: the planes of the first x are not those of the second."""
    rng = np.random.default_rng(5)
    x, w = rng.standard_normal((1536, 1280), dtype=np.float32), rng.standard_normal((1280, 1280), dtype=np.float32) / np.float32(36)
    dx, dw = (DeviceTensor.from_host(backend, t.reshape((1, 1) + t.shape)) for t in (x, w))
    first, last = (DeviceTensor.empty(backend, dx.dims) for _ in range(2))
    product = lambda out: NodeDesc(int(Op.MATMUL), out.desc, [dx.desc, dw.desc])
    backend.compute([product(first), product(dx), product(last)])
    x, w = x.astype(np.float64), w.astype(np.float64)
    for got, want in ((first, x @ w), (dx, x @ w), (last, x @ w @ w)):
        assert np.linalg.norm(got.numpy().reshape(want.shape) - want) <= 2e-5 * np.linalg.norm(want)


# an operand whose rows run backwards, so that its memory lies in front of its first element: the sum that goes there is not the product's launch's
@pytest.mark.parametrize("m,k", [(33, 33), (70, 130), (128, 1130)])
def test_results_over_an_operand_that_runs_backwards(backend, m, k):
    rng = np.random.default_rng(m + k)
    x, w, bias = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((k, k), dtype=np.float32), rng.standard_normal(k).astype(np.float32)
    results = []
    for over in (False, True):
        dx, dw, db = DeviceTensor.from_host(backend, x), DeviceTensor.from_host(backend, w.reshape(1, 1, k, k)), DeviceTensor.from_host(backend, bias)
        back = DeviceTensor(backend, dx.storage, (1, 1, m, k), (0, 0, -4 * k, 4), dx.dtype, 4 * k * (m - 1))
        prod = DeviceTensor.empty(backend, (1, 1, m, k))
        out = dx if over else DeviceTensor.empty(backend, (m, k))
        backend.compute([NodeDesc(int(Op.MATMUL), prod.desc, [back.desc, dw.desc]),
                         NodeDesc(int(Op.ADD), out.desc, [prod.reshape((m, k)).desc, db.reshape((1, k)).broadcast_to((m, k)).desc])])
        results.append(out.numpy())
    np.testing.assert_array_equal(results[1], results[0])
    want = x[::-1].astype(np.float64) @ w.astype(np.float64) + bias
    terms = np.abs(x[::-1]).astype(np.float64) @ np.abs(w).astype(np.float64) + np.abs(bias)
    assert np.all(np.abs(results[0] - want) <= (k / 8 / 4 * 2.0 ** -23 + 2.0 ** -20) * terms)
