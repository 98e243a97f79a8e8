"""The loss's kernels at the sizes where another one takes over: quads and their remainders in rows of few classes, eight threads to a row, several
blocks to an SM on long rows; every node's value against the same nodes on their own kernels."""
import numpy as np
import pytest

from test_loss_gpu import on_both

pytestmark = pytest.mark.gpu
LOG_PROBABILITIES, VALUE = 11, 16  # of the nodes' results: these, and from here on what the loss's value is made of


@pytest.mark.parametrize("rows,classes,shift", [
    (257, 31, 0), (1000, 16, 0), (131, 7, 0), (200, 32, 1), (9473, 33, 0), (9500, 127, 0), (9473, 128, 0), (9475, 129, 0), (9600, 40, 1),
    (1000, 4097, 0), (30, 8192, 0), (450, 8193, 0), (20, 16384, 0), (9, 16385, 0)])
def test_forms_of_the_loss(monkeypatch, rows, classes, shift):
    rng = np.random.default_rng(rows + classes)
    x = np.zeros(rows * classes + shift, dtype=np.float32)
    x[shift:] = 4 * rng.standard_normal(rows * classes)
    x[shift + classes:shift + 2 * classes] = -np.inf
    x[shift + 3 * classes], x[shift + 4 * classes] = np.nan, np.inf
    y = rng.integers(0, classes, rows).astype(np.int64)
    y[rows - 1] = classes - 1
    results = on_both(monkeypatch, x, y, rows, classes, shift)
    for i, (got, want) in enumerate(zip(results["1"], results["0"])):
        # a log-probability near zero is the difference of x - peak and log(sum), of up to 40 here, each rounded once and the sum in another
        # order: 40 * 2^-23 whatever the result's own size; so are those of the loss's value, and what lies between is relative to them or scaled by 1 / rows
        atol = 40 * 2.0 ** -23 if i == LOG_PROBABILITIES or i >= VALUE else 2e-6 / rows
        np.testing.assert_allclose(got, want, rtol=2e-5, atol=atol, err_msg=str(i))
