"""The single-launch kernel for small products: tile edges, K in one to eight shares, layouts, batches."""
import numpy as np
import pytest

from vkml_b200 import DeviceTensor, NodeDesc, Op

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", ["nn", "nt", "tn", "tt"])
@pytest.mark.parametrize("batch,m,k,n", [(1, 64, 784, 128), (1, 1, 1, 1), (1, 33, 127, 31), (3, 32, 128, 32), (1, 40, 129, 44), (1, 64, 260, 96),
                                         (1, 31, 1500, 65), (2, 100, 64, 10), (1, 256, 256, 256), (70, 20, 36, 24), (1, 8, 5003, 12)])
def test_small_products(backend, batch, m, k, n, layout):
    rng = np.random.default_rng(m + k + n)
    a, b = rng.standard_normal((1, batch, m, k), dtype=np.float32), rng.standard_normal((1, batch, k, n), dtype=np.float32)

    def put(x, transposed):
        return (DeviceTensor.from_host(backend, np.ascontiguousarray(np.swapaxes(x, 2, 3))).transpose(2, 3) if transposed
                else DeviceTensor.from_host(backend, x))
    da, db = put(a, layout[0] == "t"), put(b, layout[1] == "t")
    out = DeviceTensor.empty(backend, (1, batch, m, n))
    backend.set_profiling(True)
    backend.compute([NodeDesc(int(Op.MATMUL), out.desc, [da.desc, db.desc])])
    labels = [l for l, _ in backend.last_profile()]
    backend.set_profiling(False)
    assert labels == ["matmul.fp32_simt"], labels
    want = a.astype(np.float64) @ b.astype(np.float64)
    terms = np.abs(a.astype(np.float64)) @ np.abs(b.astype(np.float64))
    assert np.all(np.abs(out.numpy() - want) <= 4 * np.sqrt(k) * 2.0 ** -24 * terms + 1e-30)


# the single launch up to where more CTAs than are resident at once, a third round of K or K-slices on the tensor cores overtake it
@pytest.mark.parametrize("batch,m,k,n,small", [
    (1, 256, 256, 256, True), (1, 264, 264, 264, True), (1, 275, 376, 276, True), (1, 384, 384, 384, True), (1, 511, 256, 301, True), (1, 511, 256, 300, False),
    (1, 400, 400, 400, False), (1, 300, 484, 300, False), (1, 512, 512, 512, False), (1, 96, 784, 216, True), (1, 100, 784, 256, False),
    (32, 128, 32, 128, True), (33, 128, 32, 128, False), (8, 128, 64, 128, True), (1, 700, 33, 700, True), (1, 740, 33, 740, False)])
def test_which_products_are_small(backend, batch, m, k, n, small):
    rng = np.random.default_rng(m + k + n)
    a, b = rng.standard_normal((1, batch, m, k), dtype=np.float32), rng.standard_normal((1, batch, k, n), dtype=np.float32)
    out = DeviceTensor.empty(backend, (1, batch, m, n))
    da, db = DeviceTensor.from_host(backend, a), DeviceTensor.from_host(backend, b)
    node = NodeDesc(int(Op.MATMUL), out.desc, [da.desc, db.desc])
    assert (backend.matmul_kernel(node)[0] == "fp32_simt") == small
    backend.compute([node])
    want = a.astype(np.float64) @ b.astype(np.float64)
    terms = np.abs(a.astype(np.float64)) @ np.abs(b.astype(np.float64))
    # (the tensor cores: 22 bits per operand and a truncating accumulator of K / 8 additions per K-slice)
    bound = 4 * np.sqrt(k) * 2.0 ** -24 if small else 2.0 ** -20 + k / 8 * 2.0 ** -23
    assert np.all(np.abs(out.numpy() - want) <= bound * terms + 1e-30)
