"""The most row tiles a launch's second dimension takes, and one more: a forward
pass of 65,535 x 128 rows and of 128 more, within the 2^24 rows it accepts.
Nearly all rows are zero, so the host array is mostly untouched pages."""
import numpy as np
import pytest

import bm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [65_535 * 128, 65_535 * 128 + 1])
def test_forward_of_many_rows(rows):
    at = np.array([0, 127, 128, rows // 2, rows - 129, rows - 2, rows - 1])
    few = np.random.default_rng(1).normal(size=(len(at), bm.MLP_IN)).astype(np.float32)
    x = np.zeros((rows, bm.MLP_IN), np.float32)
    x[at] = few
    with bm.Mlp(seed=3) as net:
        y = net.forward(x)
        assert np.array_equal(y[at], net.forward(few))
        zero = net.forward(np.zeros((1, bm.MLP_IN), np.float32))[0]
    y[at] = zero
    assert (y == zero).all()
