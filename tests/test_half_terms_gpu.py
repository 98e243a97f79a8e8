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


@pytest.mark.parametrize("m,k,n,half", [(1024, 1024, 1023, False), (1024, 1024, 1024, False), (1024, 1025, 1024, True), (1000, 1433, 777, True)])
def test_from_which_size_on(backend, m, k, n, half):
    rng = np.random.default_rng(m + n)
    a, b = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((k, n), dtype=np.float32)
    got, labels = product(backend, a, b, "nn")
    assert ("matmul.tcgen05_3xf16" in labels) == half and rel(got, a, b) < 1e-5, labels


# every tile form: whole tiles and odd remainders, units for one wave and several, K-slices and none
@pytest.mark.parametrize("tile,m,k,n,layout", [
    ("256x256", 1899, 2034, 1889, "nn"), ("256x256", 2231, 1254, 1556, "tn"), ("256x256", 1000, 9001, 512, "nt"),
    ("256x128", 1086, 3267, 1052, "nt"), ("256x128", 2023, 937, 3572, "nn"), ("128x128", 1374, 1415, 1539, "nn"),
    ("128x128", 850, 2278, 2617, "nt"), ("128x128", 300, 8192, 1000, "tn"), ("128x64", 9001, 4000, 64, "nt"), ("128x64", 317, 2611, 3073, "tn")])
def test_every_tile_form(backend, tile, m, k, n, layout):
    rng = np.random.default_rng(m + k)
    a, b = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((k, n), dtype=np.float32)
    sa, sb = (DeviceTensor.empty(backend, (1, 1) + s) for s in ((m, k), (k, n)))
    out = DeviceTensor.empty(backend, (1, 1, m, n))
    name, why = backend.matmul_kernel(NodeDesc(int(Op.MATMUL), out.desc, [sa.desc, sb.desc]))
    assert name != "tcgen05_3xf16" or why.endswith(" " + tile), (name, why)
    # (twice in one span: the second one's shared planes keep a thin product from reading its operands directly)
    da, db = (DeviceTensor.from_host(backend, np.ascontiguousarray(x.T if t == "t" else x).reshape((1, 1) + (x.T if t == "t" else x).shape))
              for x, t in ((a, layout[0]), (b, layout[1])))
    da, db = (x.transpose(2, 3) if t == "t" else x for x, t in ((da, layout[0]), (db, layout[1])))
    again = DeviceTensor.empty(backend, (1, 1, m, n))
    backend.set_profiling(True)
    backend.compute([NodeDesc(int(Op.MATMUL), o.desc, [da.desc, db.desc]) for o in (out, again)])
    labels = [l for l, _ in backend.last_profile()]
    backend.set_profiling(False)
    assert labels.count("matmul.tcgen05_3xf16") == 2, labels
    assert rel(out.numpy(), a, b) < 1e-5 and same_bits(out.numpy(), again.numpy())


def test_many_products_of_changing_shapes_in_a_row(backend):
    """Sequences of odd products that change shape and tile form end, and end without a wait that ran out."""
    rng = np.random.default_rng(77)
    pool = DeviceTensor.from_host(backend, rng.standard_normal(1 << 23, dtype=np.float32))

    def matrix(rows, cols):
        return DeviceTensor(backend, pool.storage, (1, 1, rows, cols), (0, 0, cols * 4, 4), DType.F32, 0)

    for _ in range(60):
        m, n = (int(2 ** rng.uniform(7, 11.5)) | 1 for _ in range(2))
        k = min(int(4.4e9 / (2 * m * n)) + 65, (1 << 23) // max(m, n))
        out = DeviceTensor.empty(backend, (1, 1, m, n))
        right = matrix(n, k).transpose(2, 3) if rng.random() < 0.5 else matrix(k, n)
        for _ in range(30):
            backend.compute([NodeDesc(int(Op.MATMUL), out.desc, [matrix(m, k).desc, right.desc])])
    backend.synchronize()  # (raises where a bounded wait has run out)


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


@pytest.fixture(scope="module")
def tf32_backend():
    import os
    import vkml_b200
    os.environ["VKML_B200_GEMM_HALF_TERMS"] = "0"
    b = vkml_b200.Backend(0)
    del os.environ["VKML_B200_GEMM_HALF_TERMS"]
    yield b
    b.close()


def same_bits(x, y):
    return np.array_equal(np.ascontiguousarray(x).view(np.uint32), np.ascontiguousarray(y).view(np.uint32))


# K-slices where half terms have some and where they have none; 256- and 128-wide tiles; batches, one operand broadcast; odd sizes
@pytest.mark.parametrize("layout", ["nn", "nt", "tn"])
@pytest.mark.parametrize("batch,m,k,n", [(1, 512, 16384, 512), (1, 2048, 1024, 2560), (1, 1301, 1333, 1277), (5, 700, 900, 1100), (1, 260, 5000, 2500)])
def test_a_wide_operand_gets_the_tf32_product(backend, tf32_backend, batch, m, k, n, layout):
    """One element far above the others: the result is bit for bit that of TF32 terms alone, with the same tiles and K-slices."""
    rng = np.random.default_rng(batch + k)
    a, b = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((batch, k, n), dtype=np.float32)
    plain, labels = product(backend, a, b, layout)
    assert "matmul.tcgen05_3xf16" in labels
    want, labels = product(tf32_backend, a, b, layout)
    assert not any("f16" in l for l in labels) and not same_bits(plain, want)
    for at in ("a", "b"):
        wide_a, wide_b = a.copy(), b.copy()
        if at == "a":
            wide_a[m // 3, k // 2 + 1] = 3e7
        else:
            wide_b[batch // 2, k // 3, n - 1] = 3e7
        got, labels = product(backend, wide_a, wide_b, layout)
        want, _ = product(tf32_backend, wide_a, wide_b, layout)
        assert "matmul.tcgen05_3xf16" in labels and same_bits(got, want), at


# K-slices and none; batches with one operand broadcast; odd sizes
@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
@pytest.mark.parametrize("batch,m,k,n", [(1, 1536, 1280, 1280), (1, 512, 16384, 512), (5, 700, 901, 1100), (1, 1301, 1333, 1277)])
def test_strays_keep_their_share(backend, tf32_backend, batch, m, k, n, layout):
    """A few elements far below the rest, alone in their rows and columns, beside others, at one K in both operands: every
    element of the product is right beside the terms it is the sum of, from half terms."""
    rng = np.random.default_rng(m + n)
    a, b = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((batch, k, n), dtype=np.float32)
    a[5], a[6], a[m - 1] = 0, 0, 0
    b[:, :, 9], b[batch - 1, :, n - 1] = 0, 0
    tiny = np.float32(3.7e-9)
    a[5, k - 1], a[6, 3], a[6, 100], a[m - 1, 0], a[20, 3], a[20, 4] = tiny, -tiny, 2 * tiny, tiny / 1024, tiny, 1e-30
    b[:, 3, 9], b[:, 100, 9], b[batch - 1, k - 1, n - 1], b[0, 4, 33] = tiny, tiny, tiny, -tiny
    got, labels = product(backend, a, b, layout)
    assert "matmul.tcgen05_3xf16" in labels and not same_bits(got, product(tf32_backend, a, b, layout)[0])
    got = got.reshape(batch, m, n).astype(np.float64)
    a, b = a.astype(np.float64), b.astype(np.float64)
    # (an accumulator of truncating additions is off by up to K / 16 of them; both operands keep 22 bits)
    assert np.all(np.abs(got - a @ b) <= (k / 16 / 4 * 2.0 ** -23 + 2.0 ** -20) * (np.abs(a) @ np.abs(b)) + 1e-45)


@pytest.mark.parametrize("row", range(600, 608))
def test_small_elements_in_one_place(backend, tf32_backend, row):
    """More small elements than a matrix may have, all inside one piece of the sample's raster: seen in the sample or only
    by the split, the product is that of TF32 terms."""
    rng = np.random.default_rng(row)
    a, b = rng.standard_normal((2048, 2048), dtype=np.float32), rng.standard_normal((2048, 1024), dtype=np.float32)
    a[row, :100] *= np.float32(1e-12)
    assert same_bits(product(backend, a, b, "nn")[0], product(tf32_backend, a, b, "nn")[0])


def test_wide_operands_that_a_span_shares(backend, tf32_backend):
    """A layer's two backward products on a gradient of wide range, and a third on the same activations and weight: planes that stand by
    are written once and serve every product that needs them, a product of narrow operands none."""
    rng = np.random.default_rng(8)
    x, w, g = (rng.standard_normal(s, dtype=np.float32) for s in ((1536, 1152), (1152, 1280), (1536, 1280)))
    g[:, 5] *= np.exp2(rng.integers(-40, 0, 1536)).astype(np.float32)
    results = []
    for b in (backend, tf32_backend):
        def put(t):
            return DeviceTensor.from_host(b, t.reshape((1, 1) + t.shape))
        dx, dw, dg = put(x), put(w), put(g)
        outs = [DeviceTensor.empty(b, (1, 1) + s) for s in ((1152, 1280), (1536, 1152), (1536, 1280), (1280, 1280))]
        pairs = [(dx.transpose(2, 3), dg), (dg, dw.transpose(2, 3)), (dx, dw), (dg.transpose(2, 3), dg)]
        b.compute([NodeDesc(int(Op.MATMUL), o.desc, [p.desc, q.desc]) for o, (p, q) in zip(outs, pairs)])
        results.append([o.numpy() for o in outs])
    got, want = results
    assert [same_bits(p, q) for p, q in zip(got, want)] == [True, True, False, True]
    assert rel(got[2], x, w) < 6e-6


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


def test_f16_linear_layer_keeps_infinities_and_nans(backend):
    """In the fused epilogue as in separate nodes: a NaN stays one through bias and relu, an infinity keeps its sign."""
    rng = np.random.default_rng(1)
    m, k, n = 512, 256, 1024
    x, w = rng.standard_normal((m, k)).astype(np.float16), rng.standard_normal((n, k)).astype(np.float16)
    bias = rng.standard_normal(n).astype(np.float16)
    x[5, 3], x[6, 4], x[7, 200] = np.inf, np.nan, -np.inf
    bias[9], bias[10], bias[11] = np.inf, np.nan, -np.inf
    dx, dw = (DeviceTensor.from_host(backend, t.reshape((1, 1) + t.shape)) for t in (x, w))
    db = DeviceTensor.from_host(backend, bias)
    y, z, h = (DeviceTensor.empty(backend, (m, n), DType.F16) for _ in range(3))
    backend.set_profiling(True)
    backend.compute([NodeDesc(int(Op.MATMUL), y.reshape((1, 1, m, n)).desc, [dx.desc, dw.transpose(2, 3).desc]),
                     NodeDesc(int(Op.ADD), z.desc, [y.desc, db.broadcast_to((m, n)).desc]), NodeDesc(int(Op.RELU), h.desc, [z.desc])])
    labels = [l for l, _ in backend.last_profile()]
    backend.set_profiling(False)
    assert labels == ["matmul.tcgen05_f16_bias"], labels
    with np.errstate(invalid="ignore"):
        exact = x.astype(np.float64) @ w.astype(np.float64).T
        got = y.numpy()
        assert np.array_equal(np.isnan(got), np.isnan(exact)) and np.array_equal(got[5:8:2], exact[5:8:2].astype(np.float16), equal_nan=True)
        summed = (got.astype(np.float32) + bias.astype(np.float32)).astype(np.float16)
    assert np.array_equal(z.numpy(), summed, equal_nan=True)
    assert np.array_equal(h.numpy(), np.where(summed <= 0, np.float16(0), summed), equal_nan=True)
