"""A new network's tensor-core weights are those of its parameters, every time.

The parameters reach the device on the stream that converts them to bfloat16:
copied on another one, a creation in a few hundred converted weights that had
not arrived yet, and the network ranked and trained with them."""
import numpy as np
import pytest

import bm

pytestmark = pytest.mark.gpu


def test_every_new_network_is_the_same(cfg0):
    x = np.random.default_rng(1).normal(size=(128, bm.MLP_IN)).astype(np.float32)
    want = {}
    with bm.Engine.from_pair(cfg0) as E:
        for i in range(600):
            seed = i % 3
            if i % 4 == 0:   # other device work between creations
                E.set_mapping(cfg0["map0"])
                E.sweep()
            with bm.Mlp(seed=seed) as net:
                y = net.forward(x)
                if seed not in want:
                    net.set_params(net.get_params())   # converted again, long after the copy
                    want[seed] = net.forward(x)
            assert np.array_equal(y, want[seed]), (i, seed)
