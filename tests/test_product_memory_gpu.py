"""Products that are read directly run where there is no room for planes beside their operands."""
import numpy as np
import pytest

from vkml_b200 import DeviceTensor, DType, NodeDesc, Op
from vkml_b200.graph import TensorDesc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def backend():
    import vkml_b200
    b = vkml_b200.Backend(0)
    yield b
    b.close()


# (kernel for one product by itself; the addresses are only asked about)
@pytest.mark.parametrize("m,k,n,kernel", [(131072, 3072, 64, "tcgen05_3xf16"), (1048576, 1024, 64, "tcgen05_3xf16"), (1048576, 3072, 64, "tcgen05_3xtf32_direct"),
                                          (1048576, 12288, 64, "tcgen05_3xtf32_direct")])
def test_planes_that_stand_by_are_bounded(backend, m, k, n, kernel):
    a, b, out = (TensorDesc.contiguous(at << 40, (1, 1) + s, DType.F32) for at, s in ((1, (m, k)), (2, (k, n)), (3, (m, n))))
    assert backend.matmul_kernel(NodeDesc(int(Op.MATMUL), out, [a, b]))[0] == kernel


def test_a_product_runs_without_room_for_planes(backend):
    from vkml_b200.backend import OutOfMemoryError
    m, k, n = 64, 524288, 64
    rng = np.random.default_rng(1)
    x, w = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((k, n), dtype=np.float32)
    dx, dw = DeviceTensor.from_host(backend, x.reshape(1, 1, m, k)), DeviceTensor.from_host(backend, w.reshape(1, 1, k, n))
    out = DeviceTensor.empty(backend, (1, 1, m, n))
    node = NodeDesc(int(Op.MATMUL), out.desc, [dx.desc, dw.desc])
    assert backend.matmul_kernel(node)[0] == "tcgen05_3xf16"
    backend.synchronize()
    backend.trim()
    room, taken, size = backend.allocate(384 << 20), [], 64 << 30  # (the planes that stand by are 512 MB)
    while size >= 32 << 20:
        try:
            taken.append(backend.allocate(size))
        except OutOfMemoryError:
            size //= 2
    del room
    backend.trim()
    try:
        backend.compute([node])
        got = out.numpy().reshape(m, n)
    finally:
        del taken
        backend.trim()
    want, terms = x.astype(np.float64) @ w.astype(np.float64), np.abs(x).astype(np.float64) @ np.abs(w).astype(np.float64)
    chain = k / 64  # (64 slices)
    assert np.all(np.abs(got - want) <= (chain / 8 / 4 * 2.0 ** -23 + 2.0 ** -20) * terms)
