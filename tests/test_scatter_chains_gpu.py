"""scatter_add through per-destination chains: bit for bit the sums in ascending index order."""
import numpy as np
import pytest

from vkml_b200 import DeviceTensor, NodeDesc, Op, graph

pytestmark = pytest.mark.gpu


# rows of single elements and of quads, one piece and several, a ragged last piece; destinations with no, one, 32
# and 33 sources, and one that takes a third of them; long lists only, their last stretch one index or a few
@pytest.mark.parametrize("count,extent,inner", [(2100, 700, 31), (2100, 700, 129), (2100, 700, 260), (1500, 5000, 516), (700, 90, 256),
                                                (4097, 20, 256), (513, 6, 5000), (767, 12, 2052)])
def test_sums_in_index_order(backend, count, extent, inner):
    rng = np.random.default_rng(count + inner)
    idx = rng.integers(0, extent - 4, count).astype(np.int64)
    idx[rng.random(count) < 0.3] = extent - 4
    idx[rng.permutation(count)[:65]] = np.repeat([extent - 3, extent - 2], [32, 33])
    src = (rng.standard_normal((count, inner)) * 10.0 ** rng.integers(-3, 4, (count, 1))).astype(np.float32)
    want = np.zeros((extent, inner), dtype=np.float32)
    for k, j in enumerate(idx):
        want[j] += src[k]
    out = DeviceTensor.empty(backend, (extent, inner))
    srcs = [DeviceTensor.from_host(backend, src), DeviceTensor.from_host(backend, idx)]
    backend.compute([NodeDesc(int(Op.SCATTER_ADD), out.desc, [s.desc for s in srcs], graph.axis_params(0))])
    assert np.array_equal(out.numpy().view(np.uint32), want.view(np.uint32))
