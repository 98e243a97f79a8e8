"""index_select and scatter_add where their kernels change over: the width of a row, index lists with a stride, indices out of range, an axis in front."""
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


def select(b, table, index, axis):
    """The node over `index` as every second word of a longer list."""
    spread = np.full(2 * len(index), -7, np.int64)
    spread[::2] = index
    a, i = DeviceTensor.from_host(b, table), DeviceTensor.from_host(b, spread)
    i = DeviceTensor(b, i.storage, (len(index),), (16,), i.dtype)
    dims = table.shape[:axis] + (len(index),) + table.shape[axis + 1:]
    out = DeviceTensor.empty(b, dims, a.dtype)
    return out, NodeDesc(int(Op.INDEX_SELECT), out.desc, [a.desc, i.desc], graph.axis_params(axis)), (a, i)


# from one element to beyond the line between the kernels
@pytest.mark.parametrize("width", [1, 2, 5, 11, 12, 13, 31, 130])
@pytest.mark.parametrize("dtype", [np.float32, np.int64])
@pytest.mark.parametrize("axis", [0, 1])
def test_widths(backend, width, dtype, axis):
    rng = np.random.default_rng(width)
    table = rng.integers(-1000, 1000, (300, width) if axis == 0 else (3, 300, width)).astype(dtype)
    index = rng.integers(0, 300, 701)
    out, node, keep = select(backend, table, index, axis)
    backend.compute([node])
    assert np.array_equal(out.numpy(), np.take(table, index, axis))


@pytest.mark.parametrize("width", [1, 12, 33])
def test_an_index_out_of_range_is_an_error_and_clamped(backend, width):
    table = np.arange(20 * width, dtype=np.float32).reshape(20, width)
    index = np.array([3, 20, -1, 19])
    out, node, keep = select(backend, table, index, 0)
    backend.compute([node])
    with pytest.raises(IndexError):
        backend.synchronize()
    assert np.array_equal(out.numpy(), table[[3, 19, 0, 19]])


def test_narrow_rows_are_no_warp_each(backend):
    """Two million floats picked one by one take at most eight times what they take in rows of 16 (a thread to an element: twice and a half to
    three times; a warp to an element: twenty-six)."""
    rng = np.random.default_rng(3)

    def us(width):
        out, node, keep = select(backend, rng.standard_normal((4000, width), dtype=np.float32), rng.integers(0, 4000, 2_000_000 // width), 0)
        times = []
        for _ in range(6):
            backend.synchronize()
            backend.timer_begin()
            for _ in range(10):
                backend.compute([node])
            times.append(backend.timer_end())
        return min(times)
    assert us(1) < 8 * us(16)


@pytest.mark.parametrize("width", [1, 16, 33])
def test_an_empty_axis_has_no_rows_to_select(backend, width):
    a, i = DeviceTensor.empty(backend, (0, width)), DeviceTensor.from_host(backend, np.zeros(5, np.int64))
    out = DeviceTensor.empty(backend, (5, width))
    with pytest.raises(IndexError):
        backend.compute([NodeDesc(int(Op.INDEX_SELECT), out.desc, [a.desc, i.desc], graph.axis_params(0))])
    empty = DeviceTensor.empty(backend, (0, width))
    none = DeviceTensor.empty(backend, (0,), DType.I64)
    backend.compute([NodeDesc(int(Op.INDEX_SELECT), empty.desc, [a.desc, none.desc], graph.axis_params(0))])  # (none is asked for)
    backend.synchronize()


# lines of sources and chains, an axis in front of the destinations, every second word of the index list, indices out of range
@pytest.mark.parametrize("outer,extent,count,width", [(1, 500, 900, 33), (3, 500, 700, 33), (2, 40, 3000, 130), (2, (1 << 18) + 3, 900, 16)])
@pytest.mark.parametrize("beyond", [False, True])
def test_rows_are_added(backend, outer, extent, count, width, beyond):
    rng = np.random.default_rng(extent + beyond)
    src, index = rng.standard_normal((outer, count, width), dtype=np.float32), rng.integers(0, extent, count)
    index[:40] = extent - 1
    if beyond:
        index[50], index[60] = extent, -1
    spread = np.full(2 * count, -7, np.int64)
    spread[::2] = index
    s, i = DeviceTensor.from_host(backend, src), DeviceTensor.from_host(backend, spread)
    i = DeviceTensor(backend, i.storage, (count,), (16,), i.dtype)
    out = DeviceTensor.empty(backend, (outer, extent, width))
    backend.compute([NodeDesc(int(Op.SCATTER_ADD), out.desc, [s.desc, i.desc], graph.axis_params(1))])
    if beyond:
        with pytest.raises(IndexError):
            backend.synchronize()
    want = np.zeros((outer, extent, width), np.float32)
    for at, j in enumerate(index):
        if 0 <= j < extent:
            want[:, j] += src[:, at]
    assert np.array_equal(out.numpy(), want)


# every width of a task and one column more, by quads and by words, lists of all lengths
@pytest.mark.parametrize("width", [1, 32, 33, 64, 65, 127, 128, 129, 132, 257])
@pytest.mark.parametrize("extent,count", [(70, 4000), (3000, 5000)])
def test_widths_of_tasks(backend, width, extent, count):
    rng = np.random.default_rng(width)
    src = rng.standard_normal((count, width), dtype=np.float32)
    index = np.minimum(extent - 1, np.exp(rng.random(count) * np.log(extent)) - 1).astype(np.int64)  # as words of a text
    s, i, out = DeviceTensor.from_host(backend, src), DeviceTensor.from_host(backend, index), DeviceTensor.empty(backend, (extent, width))
    backend.compute([NodeDesc(int(Op.SCATTER_ADD), out.desc, [s.desc, i.desc], graph.axis_params(0))])
    want = np.zeros((extent, width), np.float32)
    for at, j in enumerate(index):
        want[j] += src[at]
    assert np.array_equal(out.numpy(), want)
