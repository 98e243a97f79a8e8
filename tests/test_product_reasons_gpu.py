"""What b200_matmul_kernel says of a product is what runs: splits inside the kernel against planes and TMA tiles."""
import numpy as np
import pytest

from vkml_b200 import DeviceTensor, NodeDesc, Op

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def backend():
    import vkml_b200
    b = vkml_b200.Backend(0)
    yield b
    b.close()


# one wave of tiles, dense (read directly before) and ragged (planes before); the streamed operand; half terms either way
@pytest.mark.parametrize("m,k,n,name,words", [
    (512, 512, 512, "tcgen05_3xtf32", "no planes"), (704, 1664, 64, "tcgen05_3xtf32_direct", "no planes"), (681, 1026, 1021, "tcgen05_3xtf32", "no planes"),
    (637, 947, 201, "tcgen05_3xtf32", "no planes"), (2400, 130, 3000, "tcgen05_3xtf32_stream", "read as fp32"),
    (512, 65536, 512, "tcgen05_3xf16", "split inside the kernel"), (1000, 1433, 777, "tcgen05_3xf16", "bound by the tensor cores"),
    (16384, 1024, 64, "tcgen05_3xtf32_direct", "")])
def test_reasons(backend, m, k, n, name, words):
    a, b = (DeviceTensor.from_host(backend, np.ones((1, 1) + s, np.float32)) for s in ((m, k), (k, n)))
    out = DeviceTensor.empty(backend, (1, 1, m, n))
    node = NodeDesc(int(Op.MATMUL), out.desc, [a.desc, b.desc])
    got, why = backend.matmul_kernel(node)
    assert (got, words in why) == (name, True), (got, why)
    if name == "tcgen05_3xf16":
        rows, columns = why.rsplit(" ", 1)[1].split("x")  # (the tile, whole)
        assert int(rows) in (128, 256) and int(columns) in (64, 128, 256), why
    backend.set_profiling(True)
    backend.compute([node])
    labels = [l for l, _ in backend.last_profile()]
    backend.set_profiling(False)
    assert "matmul." + name in labels
    if name.endswith("stream"):
        return
    inside = "no planes" in why or "split inside the kernel" in why or "fp32 tiles" in why
    assert any("split" in l for l in labels) != inside, (labels, why)


# rows along K that are read a float at a time, by both operands, one and neither: the planes' passes cost less than the first, not than the others
@pytest.mark.parametrize("m,k,n,layout,inside", [(2348, 421, 123, "nt", False), (200, 462, 2480, "nt", False), (86, 425, 2790, "nt", False),
                                                 (2348, 421, 123, "tn", True), (681, 1026, 1021, "nn", True), (637, 947, 201, "nt", True)])
def test_how_a_ragged_product_is_split(backend, m, k, n, layout, inside):
    def put(r, c, turned):
        t = DeviceTensor.from_host(backend, np.ones((1, 1) + ((c, r) if turned else (r, c)), np.float32))
        return t.transpose(2, 3) if turned else t
    a, b, out = put(m, k, layout[0] == "t"), put(k, n, layout[1] == "t"), DeviceTensor.empty(backend, (1, 1, m, n))
    why = backend.matmul_kernel(NodeDesc(int(Op.MATMUL), out.desc, [a.desc, b.desc]))[1]
    assert ("inside the kernel" in why) == inside, why
