"""Padded rows add nothing to the gradients, whatever the weights make of them.

Hidden unit 0 is 0 on every real row and 2^127 on a zero row, so the second
layer is infinite on the padding and finite on the real rows."""
import numpy as np
import pytest

import bm
import mlp_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 127, 129])
def test_infinite_activations_of_padded_rows(rows):
    rng = np.random.default_rng(rows)
    p = mo.init_params(rows).astype(np.float32)
    q = mo.unpack(p)
    q["W1"][0] = 0
    q["W1"][0, 0] = -2.0 ** 127
    q["b1"][0] = 2.0 ** 127
    q["W2"][:, 0] = 4
    p = np.concatenate([q[k].ravel() for k, _ in mo.SIZES]).astype(np.float32)
    x = rng.normal(size=(rows, mo.IN)).astype(np.float32)
    x[:, 0] = 1
    t = rng.normal(size=rows).astype(np.float32)
    with bm.Mlp(seed=1) as net:
        net.set_params(p)
        loss, g = net.train_step(x, t, lr=0.0)
    # on the real rows unit 0 is 0: the network without it
    r = mo.unpack(p.copy())
    r["W1"][0] = r["b1"][0] = 0
    r["W2"][:, 0] = 0
    want_loss, want = mo.forward_backward(np.concatenate([r[k].ravel() for k, _ in mo.SIZES]), x, t, bf16_path=True)
    assert np.isfinite(g).all()
    assert abs(loss - want_loss) <= 1e-3 * max(1.0, want_loss)
    # 2e-3 in the 2-norm: the tolerance of the network's other gradient tests
    for name in ("b1", "W2", "b2", "w3", "b3"):
        a, b = mo.unpack(g)[name], mo.unpack(want)[name]
        assert np.linalg.norm(a - b) <= 2e-3 * np.linalg.norm(b) + 1e-7, name
