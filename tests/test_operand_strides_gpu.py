"""The kernels that read a product's operands themselves, over views of every kind: pitches wider than a row, beginnings off 16 bytes, two batch axes
or one of them standing still, axes that stand still or run backwards, no axis of unit stride; with strays and with an operand that half terms cannot
hold, whose places are counted in such a view.  Against float64."""
import os

import numpy as np
import pytest

from vkml_b200 import DeviceTensor, DType, NodeDesc, Op

pytestmark = pytest.mark.gpu


def context(**switches):
    import vkml_b200
    for key, value in switches.items():
        os.environ["VKML_B200_GEMM_" + key] = value
    b = vkml_b200.Backend(0)
    for key in switches:
        del os.environ["VKML_B200_GEMM_" + key]
    return b


@pytest.fixture(scope="module")
def half_terms():
    b = context(INLINE="1")
    yield b
    b.close()


@pytest.fixture(scope="module")
def tf32_terms():
    b = context(INLINE="8", STREAM="0")
    yield b
    b.close()


def layout(form, batch, r, c):
    """Element strides over (b0, b1, r, c), the first element's place and how many elements the buffer has."""
    b0, b1 = batch
    strides = {"dense": (c, 1), "pitch": (c + 5, 1), "quads": (c + 8, 1), "turned": (1, r), "turned pitch": (1, r + 3), "turned quads": (1, r + 4),
               "no unit": (2 * c + 3, 2), "rows still": (0, 1), "columns still": (1, 0), "backwards": (-(c + 1), 1), "turned backwards": (1, -(r + 4)),
               "both one": (1, 1)}[form.split("+")[0]]
    reach = [(e - 1) * s for e, s in zip((r, c), strides)]
    start, size = -sum(x for x in reach if x < 0), sum(abs(x) for x in reach) + 1
    step = (size + 3) // 4 * 4 + (1 if "odd" in form else 0)  # (batches that do not begin on 16 bytes)
    s_b1 = 0 if "inner still" in form else step
    s_b0 = 0 if "outer still" in form else step * (b1 if s_b1 else 1)
    start += 3 if "offset" in form else 0
    return (s_b0, s_b1) + strides, start, start + size + (b0 - 1) * s_b0 + (b1 - 1) * s_b1


def operand(backend, form, batch, r, c, dtype, rng, touch=lambda flat: None):
    strides, start, size = layout(form, batch, r, c)
    flat = rng.standard_normal(size + 8).astype(dtype)
    touch(flat)
    t = DeviceTensor.from_host(backend, flat)
    w = flat.itemsize
    dims = batch + (r, c)
    view = np.lib.stride_tricks.as_strided(flat[start:], dims, [s * w for s in strides], writeable=False)
    return DeviceTensor(backend, t.storage, dims, [s * w for s in strides], t.dtype, start * w), view


def product(backend, a, b, dtype):
    out = DeviceTensor.empty(backend, a.dims[:3] + b.dims[3:], dtype)
    backend.set_profiling(True)
    backend.compute([NodeDesc(int(Op.MATMUL), out.desc, [a.desc, b.desc])])
    labels = [l for l, _ in backend.last_profile()]
    backend.set_profiling(False)
    return out.numpy().astype(np.float64), labels


FORMS = ["pitch", "quads", "dense+offset", "turned", "turned pitch", "turned quads", "turned+offset", "no unit", "rows still", "columns still", "backwards",
         "turned backwards", "both one"]
BATCHES = ["dense", "dense+outer still", "dense+inner still", "dense+odd", "turned+odd+inner still", "pitch+outer still+inner still"]
CASES = [(f, "dense", (1, 1)) for f in FORMS] + [("turned", f, (1, 1)) for f in FORMS] + [(f, "quads", (2, 3)) for f in BATCHES] + [("pitch", f, (2, 3)) for f in BATCHES]
SIZES = [(197, 517, 333), (196, 516, 332)]


@pytest.mark.parametrize("m,k,n", SIZES)
@pytest.mark.parametrize("fa,fb,batch", CASES)
@pytest.mark.parametrize("terms", ["half", "tf32"])
def test_fp32(request, terms, fa, fb, batch, m, k, n):
    backend = request.getfixturevalue(terms + "_terms")
    rng = np.random.default_rng(m + len(fa) + len(fb))
    (da, a), (db, b) = operand(backend, fa, batch, m, k, "f4", rng), operand(backend, fb, batch, k, n, "f4", rng)
    got, labels = product(backend, da, db, DType.F32)
    assert not any("split" in l for l in labels) and any("tcgen05" in l for l in labels), labels
    a, b = a.astype(np.float64), b.astype(np.float64)
    step = 16 if terms == "half" else 8  # of K in one addition to an accumulator
    assert np.all(np.abs(got - a @ b) <= (k / step / 4 * 2.0 ** -23 + 2.0 ** -20) * (np.abs(a) @ np.abs(b)) + 1e-45)


# an element too small beside the rest (left out and added back), one too large (planes stand by), rows of nothing else beside them
@pytest.mark.parametrize("kind", ["stray", "wide"])
@pytest.mark.parametrize("fa,fb,batch", [("pitch", "turned pitch", (1, 1)), ("no unit", "backwards", (1, 1)), ("turned backwards", "dense+offset", (1, 1)),
                                         ("dense+inner still", "turned+odd", (2, 3)), ("turned+odd+outer still", "quads+inner still", (2, 3))])
def test_ranges(half_terms, kind, fa, fb, batch):
    m, k, n = SIZES[0]
    rng = np.random.default_rng(len(fa))

    def touch(flat):
        at = rng.integers(0, flat.size, 5)
        flat[at] = np.float32(3.7e-9) if kind == "stray" else np.float32(1e9)
    (da, a), (db, b) = operand(half_terms, fa, batch, m, k, "f4", rng, touch), operand(half_terms, fb, batch, k, n, "f4", rng)
    got, labels = product(half_terms, da, db, DType.F32)
    a, b = a.astype(np.float64), b.astype(np.float64)
    assert np.all(np.abs(got - a @ b) <= (k / 8 / 4 * 2.0 ** -23 + 2.0 ** -20) * (np.abs(a) @ np.abs(b)) + 1e-45)


@pytest.mark.parametrize("m,k,n", SIZES)
@pytest.mark.parametrize("fa,fb,batch", CASES)
def test_half_storage(half_terms, fa, fb, batch, m, k, n):
    rng = np.random.default_rng(m + len(fa) + len(fb))
    (da, a), (db, b) = operand(half_terms, fa, batch, m, k, "f2", rng), operand(half_terms, fb, batch, k, n, "f2", rng)
    got, labels = product(half_terms, da, db, DType.F16)
    want = a.astype(np.float64) @ b.astype(np.float64)
    ulp = np.spacing(np.abs(want).astype(np.float16)).astype(np.float64)
    assert np.all(np.abs(got - want) <= 0.5 * ulp + 1e-5 * np.sqrt(k))
    if "no unit" not in (fa, fb):
        assert "f16.widen" not in labels, labels
