"""Half-storage products whose rows lie anywhere: odd and even pitches, every layout, tile edges, K that ends inside a stage, K-slices, batches, and
Linear layers with bias and relu, against float64."""
import numpy as np
import pytest

from vkml_b200 import DeviceTensor, DType, NodeDesc, Op

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def backend():
    import vkml_b200
    b = vkml_b200.Backend(0)
    yield b
    b.close()


def run(backend, nodes):
    backend.set_profiling(True)
    backend.compute(nodes)
    labels = [l for l, _ in backend.last_profile()]
    backend.set_profiling(False)
    return labels


def close(got, a, b):
    """One rounding to half, and the fp32 accumulator's error where it decides between neighbours."""
    want = a.astype(np.float64) @ b.astype(np.float64)
    ulp = np.spacing(np.abs(want).astype(np.float16)).astype(np.float64)
    assert np.all(np.abs(got.reshape(want.shape).astype(np.float64) - want) <= 0.5 * ulp + 1e-5 * np.sqrt(a.shape[-1]))


# one tile and its neighbours, a pair's tiles, one row or column too many, K of a part of a stage and one more than one, slices, batches
@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
@pytest.mark.parametrize("batch,m,k,n", [(1, 130, 129, 2050), (1, 247, 348, 1130), (1, 2049, 65, 2301), (1, 33, 4098, 270), (1, 513, 62, 1031), (3, 257, 301, 219),
                                         (1, 1500, 518, 1602)])
def test_products_of_any_pitch(backend, batch, m, k, n, layout):
    rng = np.random.default_rng(m + k + n)
    a, b = rng.standard_normal((m, k)).astype(np.float16), rng.standard_normal((batch, k, n)).astype(np.float16)

    def put(x, transposed):
        x = np.ascontiguousarray(np.swapaxes(x, -1, -2)) if transposed else np.ascontiguousarray(x)
        t = DeviceTensor.from_host(backend, x.reshape((1,) * (4 - x.ndim) + x.shape))
        return t.transpose(2, 3) if transposed else t
    da, db = put(a, layout[0] == "t"), put(b, layout[1] == "t")
    da, db = (t.broadcast_to((1, batch) + t.dims[2:]) for t in (da, db))
    out = DeviceTensor.empty(backend, (1, batch, m, n), DType.F16)
    labels = run(backend, [NodeDesc(int(Op.MATMUL), out.desc, [da.desc, db.desc])])
    assert "matmul.tcgen05_f16" in labels and "f16.widen" not in labels, labels
    close(out.numpy(), a, b)


def test_an_operand_that_begins_on_an_odd_half(backend):
    rng = np.random.default_rng(3)
    a, b = rng.standard_normal((300, 402)).astype(np.float16), rng.standard_normal((400, 512)).astype(np.float16)
    da, db = DeviceTensor.from_host(backend, a), DeviceTensor.from_host(backend, b.reshape(1, 1, 400, 512))
    view = DeviceTensor(backend, da.storage, (1, 1, 300, 400), (0, 0, 804, 2), DType.F16, 2)
    out = DeviceTensor.empty(backend, (1, 1, 300, 512), DType.F16)
    labels = run(backend, [NodeDesc(int(Op.MATMUL), out.desc, [view.desc, db.desc])])
    assert "matmul.tcgen05_f16" in labels, labels
    close(out.numpy(), a[:, 1:401], b)


# the epilogue's own addition and the fold's; the narrowest result; relu and none; infinities and NaNs
@pytest.mark.parametrize("relu", [False, True])
@pytest.mark.parametrize("m,k,n", [(247, 348, 1369), (2049, 130, 2301), (40, 4099, 300), (64, 2100, 257)])
def test_linear_layers_of_any_pitch(backend, m, k, n, relu):
    rng = np.random.default_rng(m + n)
    x, w = rng.standard_normal((m, k)).astype(np.float16), rng.standard_normal((n, k)).astype(np.float16)
    bias = (8 * rng.standard_normal(n)).astype(np.float16)
    x[5, 3], x[6, 4], bias[9], bias[10] = np.inf, np.nan, -np.inf, np.nan
    dx, dw = (DeviceTensor.from_host(backend, t.reshape((1, 1) + t.shape)) for t in (x, w))
    db = DeviceTensor.from_host(backend, bias)
    y, z, h = (DeviceTensor.empty(backend, (m, n), DType.F16) for _ in range(3))
    nodes = [NodeDesc(int(Op.MATMUL), y.reshape((1, 1, m, n)).desc, [dx.desc, dw.transpose(2, 3).desc]),
             NodeDesc(int(Op.ADD), z.desc, [y.desc, db.broadcast_to((m, n)).desc])]
    if relu:
        nodes.append(NodeDesc(int(Op.RELU), h.desc, [z.desc]))
    labels = run(backend, nodes)
    assert "matmul.tcgen05_f16_bias" in labels and set(labels) <= {"matmul.tcgen05_f16_bias", "matmul.fold"}, labels
    got = y.numpy()
    keep = [i for i in range(m) if i not in (5, 6)]
    close(got[keep], x[keep], w.T)
    with np.errstate(invalid="ignore"):
        assert np.array_equal(np.isnan(got), np.isnan(x.astype(np.float64) @ w.astype(np.float64).T))
        summed = (got.astype(np.float32) + bias.astype(np.float32)).astype(np.float16)
    assert np.array_equal(z.numpy(), summed, equal_nan=True)
    if relu:
        assert np.array_equal(h.numpy(), np.where(summed <= 0, np.float16(0), summed), equal_nan=True)
