"""The kind::f16 tensor-core kernel: F32 products from two half terms per operand (with the TF32 planes that
stand by for operands of a wide range), and F16 storage, against float64."""
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


def product(backend, a, b, layout):
    """a[.., m, k] . b[.., k, n], the operands stored as `layout` says (t: transposed); result and kernels."""
    def put(x, transposed):
        x = np.ascontiguousarray(np.swapaxes(x, -1, -2)) if transposed else np.ascontiguousarray(x)
        t = DeviceTensor.from_host(backend, x.reshape((1,) * (4 - x.ndim) + x.shape))
        return t.transpose(2, 3) if transposed else t
    da, db = put(a, layout[0] == "t"), put(b, layout[1] == "t")
    batch = max(da.dims[1], db.dims[1])
    da, db = (t.broadcast_to((1, batch) + t.dims[2:]) for t in (da, db))
    out = DeviceTensor.empty(backend, (1, batch, da.dims[2], db.dims[3]), da.dtype)
    backend.set_profiling(True)
    backend.compute([NodeDesc(int(Op.MATMUL), out.desc, [da.desc, db.desc])])
    labels = [l for l, _ in backend.last_profile()]
    backend.set_profiling(False)
    return out.numpy(), labels


def rel(got, a, b):
    want = a.astype(np.float64) @ b.astype(np.float64)
    return np.linalg.norm(got.reshape(want.shape).astype(np.float64) - want) / np.linalg.norm(want)


# whole tiles; ragged in every extent with odd pitches; a last tile of one row and column; K-slices; batches
# with a broadcast operand; a last K-block of one
@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
@pytest.mark.parametrize("m,k,n", [(1536, 1280, 1280), (1301, 1333, 1277), (1025, 2049, 1281), (300, 8193, 1000)])
def test_f32_products_from_half_terms(backend, m, k, n, layout):
    rng = np.random.default_rng(m + k)
    a, b = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((k, n), dtype=np.float32)
    got, labels = product(backend, a, b, layout)
    assert "matmul.tcgen05_3xf16" in labels, labels
    assert rel(got, a, b) < 6e-6


def test_batches_and_a_broadcast_operand(backend):
    rng = np.random.default_rng(5)
    a, b = rng.standard_normal((9, 500, 516), dtype=np.float32), rng.standard_normal((516, 1030), dtype=np.float32)
    got, labels = product(backend, a, b, "nn")
    assert "matmul.tcgen05_3xf16" in labels and rel(got, a, b) < 6e-6


@pytest.mark.parametrize("kind", ["outlier", "spread", "tiny rows", "inf", "nan", "subnormal", "zero"])
def test_ranges(backend, kind):
    """Operands that two half terms cannot hold take the TF32 planes: nothing is lost beside what those lose."""
    rng = np.random.default_rng(17)
    a = rng.standard_normal((1400, 1300), dtype=np.float32)
    b = rng.standard_normal((1300, 1300), dtype=np.float32)
    if kind == "outlier":    # one element far above any sample
        a[700, 701] = 1e9
    elif kind == "spread":   # 2^-30 .. 2^30 everywhere
        a *= np.exp2(rng.integers(-30, 30, a.shape)).astype(np.float32)
    elif kind == "tiny rows":  # rows of their own scale: each has to be right beside itself
        a[100:140] *= np.float32(1e-12)
    elif kind == "inf":
        a[3, 5] = np.inf
    elif kind == "nan":
        b[5, 7] = np.nan
    elif kind == "subnormal":
        a *= np.float32(1e-41)
        b *= np.float32(1e10)
    elif kind == "zero":
        a[:] = 0
    got, _ = product(backend, a, b, "nn")
    got = got.reshape(1400, 1300)
    if kind == "zero":
        assert np.array_equal(got, np.zeros_like(got))
        return
    if kind in ("inf", "nan"):
        bad = np.zeros_like(got, dtype=bool)
        bad[3 if kind == "inf" else slice(None), slice(None) if kind == "inf" else 7] = True
        assert np.array_equal(~np.isfinite(got), bad)
        return
    want = a.astype(np.float64) @ b.astype(np.float64)
    rows = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
    assert rows.max() < 2e-5, rows.max()


@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
@pytest.mark.parametrize("m,k,n", [(256, 256, 256), (264, 520, 264), (104, 336, 776), (64, 4096, 512), (40, 1024, 1000)])
def test_f16_storage_products(backend, m, k, n, layout):
    rng = np.random.default_rng(m + k + n)
    a, b = rng.standard_normal((m, k)).astype(np.float16), rng.standard_normal((k, n)).astype(np.float16)
    got, labels = product(backend, a, b, layout)
    assert got.dtype == np.float16 and "matmul.tcgen05_f16" in labels, labels
    want = a.astype(np.float64) @ b.astype(np.float64)
    ulp = np.spacing(np.abs(want).astype(np.float16)).astype(np.float64)
    err = np.abs(got.reshape(want.shape).astype(np.float64) - want)
    # one rounding to half, and the fp32 accumulator's error where it decides between neighbours
    assert np.all(err <= 0.5 * ulp + 1e-5 * np.sqrt(k))


# a tile and its remainder in rows, one pair of accumulators and several, with and without the relu; sizes that keep the nodes apart
@pytest.mark.parametrize("relu", [False, True])
@pytest.mark.parametrize("m,k,n", [(300, 512, 4096), (1023, 256, 1088), (2048, 64, 1024), (200, 512, 1000)])
def test_f16_linear_layers(backend, m, k, n, relu):
    rng = np.random.default_rng(m + n)
    x, w = rng.standard_normal((m, k)).astype(np.float16), rng.standard_normal((n, k)).astype(np.float16)
    bias = (8 * rng.standard_normal(n)).astype(np.float16)
    dx, dw = (DeviceTensor.from_host(backend, t.reshape((1, 1) + t.shape)) for t in (x, w))
    y, z, h = (DeviceTensor.empty(backend, (m, n), DType.F16) for _ in range(3))
    nodes = [NodeDesc(int(Op.MATMUL), y.reshape((1, 1, m, n)).desc, [dx.desc, dw.transpose(2, 3).desc]),
             NodeDesc(int(Op.ADD), z.desc, [y.desc, DeviceTensor.from_host(backend, bias).broadcast_to((m, n)).desc])]
    if relu:
        nodes.append(NodeDesc(int(Op.RELU), h.desc, [z.desc]))
    keep = DeviceTensor.from_host(backend, bias)
    nodes[1].src[1] = keep.broadcast_to((m, n)).desc
    backend.compute(nodes)
    got = y.numpy()
    want = x.astype(np.float64) @ w.astype(np.float64).T
    assert np.all(np.abs(got - want) <= 0.5 * np.spacing(np.abs(want).astype(np.float16)).astype(np.float64) + 1e-5 * np.sqrt(k))
    summed = (got.astype(np.float32) + bias.astype(np.float32)).astype(np.float16)
    assert np.array_equal(z.numpy().view(np.uint16), summed.view(np.uint16))
    if relu:
        assert np.array_equal(h.numpy(), np.where(summed <= 0, np.float16(0), summed))
