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
    import torch
    b = context("8")  # (TF32 terms inside the kernel wherever they fit)
    m, k, n = 300, 1024, 72
    rng = np.random.default_rng(pitch)
    x, w = rng.standard_normal((m, k), dtype=np.float32), rng.standard_normal((n, k), dtype=np.float32)
    dx, wide = DeviceTensor.from_host(b, x.reshape(1, 1, m, k)), DeviceTensor.empty(b, (n, pitch))
    b.synchronize()
    face = type("Face", (), {"__cuda_array_interface__": {"shape": (n, pitch), "typestr": "<f4", "data": (wide.desc.data, False), "strides": None, "version": 3}})()
    torch.as_tensor(face, device="cuda")[:, :k] = torch.from_numpy(w).cuda()
    torch.cuda.synchronize()
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
