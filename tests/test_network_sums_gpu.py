"""The weight gradients are sums over all rows in one order: the same call gives
the same bits.  (Bias and output-layer gradients add a block's rows with float
atomics and may differ in the last bits.)"""
import numpy as np
import pytest

import bm
import mlp_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1024, 1536, 2100, 8000])
def test_weight_gradients_repeat(rows):
    rng = np.random.default_rng(rows)
    p = mo.init_params(rows).astype(np.float32)
    x = rng.normal(size=(rows, mo.IN)).astype(np.float32)
    t = rng.normal(size=rows).astype(np.float32)
    with bm.Mlp(seed=1) as net:
        net.set_params(p)
        first = mo.unpack(net.train_step(x, t, lr=0.0)[1])
        for _ in range(5):
            again = mo.unpack(net.train_step(x, t, lr=0.0)[1])
            for name in ("W1", "W2"):
                assert np.array_equal(first[name], again[name]), name
