"""Bias, mask and relu as one launch at sizes that are no multiple of a quad, the relu next to its add or behind other nodes."""
import numpy as np
import pytest

from vkml_b200 import DeviceTensor, DType, NodeDesc, Op, graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("late", [False, True])
@pytest.mark.parametrize("dims,axis", [((64, 128), 1), ((31, 161), 1), ((3, 2), 1), ((7, 5, 3, 3), 1), ((2, 6, 4, 4), 1), ((5, 7, 15, 15), 1)])
def test_bias_mask_relu(backend, dims, axis, late):
    rng = np.random.default_rng(sum(dims))
    x, bias = rng.standard_normal(dims).astype(np.float32), rng.standard_normal(dims[axis]).astype(np.float32)
    x.reshape(-1)[0] = np.nan
    dx, db = DeviceTensor.from_host(backend, x), DeviceTensor.from_host(backend, bias)
    wide = tuple(dims[axis] if i == axis else 1 for i in range(len(dims)))
    y, a, b, relu, other = (DeviceTensor.empty(backend, dims) for _ in range(5))
    mask = DeviceTensor.empty(backend, dims, DType.BOOL)
    full = graph.full_params(0.0)
    nodes = [NodeDesc(int(Op.ADD), y.desc, [dx.desc, db.reshape(wide).broadcast_to(dims).desc]), NodeDesc(int(Op.FULL), a.desc, [], full),
             NodeDesc(int(Op.LESS_EQUAL), mask.desc, [y.desc, a.desc]), NodeDesc(int(Op.FULL), b.desc, [], full)]
    tail = [NodeDesc(int(Op.RELU), relu.desc, [y.desc])]
    between = [NodeDesc(int(Op.EXP), other.desc, [dx.desc])]
    backend.set_profiling(True)
    backend.compute(nodes + (between + tail if late else tail + between))
    labels = [l for l, _ in backend.last_profile()]
    backend.set_profiling(False)
    assert labels == ["fused.bias_mask_relu", "exp"], labels
    want = x + bias.reshape(wide)
    np.testing.assert_array_equal(y.numpy(), want)
    np.testing.assert_array_equal(mask.numpy(), (want <= 0).astype(np.uint8))
    np.testing.assert_array_equal(relu.numpy(), np.where(want <= 0, np.float32(0), want))
    assert not a.numpy().any() and not b.numpy().any()
