"""TF32 terms split inside the kernel give, bit for bit, what TF32 planes give: every layout, tile edges, a K that ends inside a stage, K-slices,
batches, values past the range."""
import os

import numpy as np
import pytest

from vkml_b200 import DeviceTensor, NodeDesc, Op

pytestmark = pytest.mark.gpu


def context(value):
    import vkml_b200
    os.environ["VKML_B200_GEMM_INLINE"] = value
    b = vkml_b200.Backend(0)
    del os.environ["VKML_B200_GEMM_INLINE"]
    return b


@pytest.fixture(scope="module")
def backends():
    pair = context("auto"), context("0")
    yield pair
    for b in pair:
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
    return out.numpy(), labels


# one row or column more or less than a tile; narrow results; K of a part of a stage and one more than a stage; slices; whole quads and none; batches
@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
@pytest.mark.parametrize("batch,m,k,n", [(1, 512, 512, 512), (1, 300, 1001, 257), (1, 129, 1537, 385), (1, 641, 947, 63), (1, 68, 838, 389), (1, 1030, 33, 1010),
                                         (3, 257, 301, 219), (1, 33, 4099, 301), (1, 640, 2176, 128)])
def test_the_same_bits_as_from_planes(backends, batch, m, k, n, layout):
    rng = np.random.default_rng(m + k + n)
    a, b = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((batch, k, n), dtype=np.float32)
    got, labels = product(backends[0], a, b, layout)
    want, others = product(backends[1], a, b, layout)
    main = {"matmul.tcgen05_3xtf32", "matmul.tcgen05_3xtf32_direct"}
    if main & set(labels):  # (a layout whose right operand streams stays with that kernel)
        assert not any("split" in l for l in labels), labels
    assert labels.count("matmul.fold") == others.count("matmul.fold")
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("m,k,n", [(512, 512, 512), (301, 1003, 259)])
def test_values_past_the_range(backends, m, k, n):
    rng = np.random.default_rng(m)
    a, b = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((k, n), dtype=np.float32)
    a[1, 5], a[2, 6], a[3, 7], a[4, k - 1] = np.inf, np.nan, 3.4028e38, -np.inf
    a[5] *= np.float32(1e-41)
    b[9, 4] = np.float32(-3.4028235e38)
    got, want = (product(x, a, b, "nn")[0] for x in backends)
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
