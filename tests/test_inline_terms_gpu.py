"""Products whose operands are split into half terms inside the kernel, against float64: every layout, tile edges, a K that ends inside a
stage, batches, strays and operands that half terms cannot hold."""
import os

import numpy as np
import pytest

from vkml_b200 import DeviceTensor, NodeDesc, Op

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def backend():
    import vkml_b200
    os.environ["VKML_B200_GEMM_INLINE"] = "1"
    b = vkml_b200.Backend(0)
    del os.environ["VKML_B200_GEMM_INLINE"]
    yield b
    b.close()


def product(backend, a, b, layout):
    def put(x, transposed):
        x = np.ascontiguousarray(np.swapaxes(x, -1, -2)) if transposed else np.ascontiguousarray(x)
        t = DeviceTensor.from_host(backend, x.reshape((1,) * (4 - x.ndim) + x.shape))
        return t.transpose(2, 3) if transposed else t
    da, db = put(a, layout[0] == "t"), put(b, layout[1] == "t")
    batch = max(da.dims[1], db.dims[1])
    da, db = (t.broadcast_to((1, batch) + t.dims[2:]) for t in (da, db))
    out = DeviceTensor.empty(backend, (1, batch, da.dims[2], db.dims[3]))
    backend.set_profiling(True)
    backend.compute([NodeDesc(int(Op.MATMUL), out.desc, [da.desc, db.desc])])
    labels = [l for l, _ in backend.last_profile()]
    backend.set_profiling(False)
    assert "matmul.tcgen05_3xf16" in labels and "matmul.split" not in labels, labels
    return out.numpy()


def check(got, a, b):
    """22 bits in each operand, and an accumulator that truncates K / 16 additions."""
    a, b = a.astype(np.float64), b.astype(np.float64)
    want, terms = a @ b, np.abs(a) @ np.abs(b)
    k = a.shape[-1]
    assert np.all(np.abs(got.reshape(want.shape) - want) <= (k / 16 / 4 * 2.0 ** -23 + 2.0 ** -20) * terms + 1e-45)


# the pair's tile and the narrow one, by extents; whole quads and none; one row or column more than a tile; an odd CTA without rows;
# K of a part of a stage, one more than a stage, many slices; several tiles to a pair
@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
@pytest.mark.parametrize("batch,m,k,n", [(1, 256, 512, 256), (1, 257, 513, 259), (1, 384, 132, 520), (1, 100, 4096, 300), (1, 33, 2049, 1027), (1, 640, 1000, 64),
                                         (3, 130, 260, 516), (2, 1000, 65, 700), (90, 256, 64, 256), (1, 512, 16388, 260)])
def test_inline_products(backend, batch, m, k, n, layout):
    rng = np.random.default_rng(m + k + n)
    a, b = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((batch, k, n), dtype=np.float32)
    check(product(backend, a, b, layout), a, b)


@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
@pytest.mark.parametrize("batch,m,k,n", [(1, 300, 1000, 260), (2, 257, 777, 515), (1, 64, 4096, 512)])
def test_inline_strays_keep_their_share(backend, batch, m, k, n, layout):
    rng = np.random.default_rng(m + n)
    a, b = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((batch, k, n), dtype=np.float32)
    a[5], a[m - 1], b[:, :, 9], b[batch - 1, :, n - 1] = 0, 0, 0, 0
    tiny = np.float32(3.7e-9)
    a[5, k - 1], a[5, 3], a[m - 1, 0], a[20, 3], a[20, 4] = tiny, -tiny, tiny / 1024, tiny, 1e-30
    b[:, 3, 9], b[batch - 1, k - 1, n - 1], b[0, 4, 33] = tiny, tiny, -tiny
    check(product(backend, a, b, layout), a, b)


@pytest.mark.parametrize("kind", ["outlier", "spread", "tiny rows", "inf", "nan", "subnormal", "large", "zero"])
def test_inline_ranges(backend, kind):
    rng = np.random.default_rng(17)
    a, b = rng.standard_normal((700, 650), dtype=np.float32), rng.standard_normal((650, 520), dtype=np.float32)
    if kind == "outlier":
        a[350, 351] = 1e9
    elif kind == "spread":
        a *= np.exp2(rng.integers(-30, 30, a.shape)).astype(np.float32)
    elif kind == "tiny rows":
        a[100:140] *= np.float32(1e-12)
    elif kind == "inf":
        a[3, 5] = np.inf
    elif kind == "nan":
        b[5, 7] = np.nan
    elif kind == "subnormal":
        a, b = a * np.float32(1e-41), b * np.float32(1e10)
    elif kind == "large":
        a, b = a * np.float32(1e30), b * np.float32(1e-25)
    elif kind == "zero":
        a[:] = 0
    got = product(backend, a, b, "nn").reshape(700, 520)
    if kind in ("inf", "nan"):
        bad = np.zeros_like(got, dtype=bool)
        bad[3 if kind == "inf" else slice(None), slice(None) if kind == "inf" else 7] = True
        assert np.array_equal(~np.isfinite(got), bad)
        return
    want = a.astype(np.float64) @ b.astype(np.float64)
    assert np.all(np.linalg.norm(got - want, axis=1) <= 2e-5 * np.linalg.norm(want, axis=1))
