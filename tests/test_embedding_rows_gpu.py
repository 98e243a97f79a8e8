"""index_select and scatter_add on rows that are no quads: widths around a warp's pieces, 4- and 8-byte elements, lists of one, a few and many
sources, a destination axis too long for a line of sources each; against numpy, bit for bit (sums in index order)."""
import numpy as np
import pytest

from vkml_b200 import DeviceTensor, DType, NodeDesc, Op, graph

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def backend():
    import vkml_b200
    b = vkml_b200.Backend(0)
    yield b
    b.close()


@pytest.mark.parametrize("width", [1, 31, 33, 64, 65, 127, 129, 255, 257, 483])
@pytest.mark.parametrize("dtype", [np.float32, np.int64])
def test_rows_are_selected(backend, width, dtype):
    rng = np.random.default_rng(width)
    table, index = rng.integers(-1000, 1000, (700, width)).astype(dtype), rng.integers(0, 700, 1301)
    a, i = DeviceTensor.from_host(backend, table), DeviceTensor.from_host(backend, index)
    out = DeviceTensor.empty(backend, (1301, width), a.dtype)
    backend.compute([NodeDesc(int(Op.INDEX_SELECT), out.desc, [a.desc, i.desc], graph.axis_params(0))])
    assert np.array_equal(out.numpy(), table[index])


# one source each, a few, more than 32 (found by reading the list), and destinations beyond the lines' reach
@pytest.mark.parametrize("extent,count,width", [(5000, 600, 83), (3000, 9000, 129), (2000, 6000, 483), (40, 3000, 257), (300, 3000, 130), (1500, 4001, 512),
                                                ((1 << 18) + 7, 2000, 33)])
def test_rows_are_added_in_index_order(backend, extent, count, width):
    rng = np.random.default_rng(extent + width)
    src, index = rng.standard_normal((count, width), dtype=np.float32), rng.integers(0, extent, count)
    index[:5] = extent - 1
    s, i = DeviceTensor.from_host(backend, src), DeviceTensor.from_host(backend, index)
    out = DeviceTensor.empty(backend, (extent, width))
    backend.compute([NodeDesc(int(Op.SCATTER_ADD), out.desc, [s.desc, i.desc], graph.axis_params(0))])
    want = np.zeros((extent, width), np.float32)
    for k, j in enumerate(index):
        want[j] += src[k]
    assert np.array_equal(out.numpy(), want)
