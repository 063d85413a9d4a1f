"""The network's kernels at the edges of their tiles: training rows that end in
and behind a 512-row share of the weight gradients' split sums, and ranked
pairs that end in a tile of 128, in the first and second tile of each SM and
behind them.

Tolerances as derived for the network's other tests: the CUDA path and the
oracle's bf16 form round the same values to bfloat16 and accumulate in float32,
so they differ by summation order and the rare bf16 rounding it flips: 2e-3
relative for gradients in the 2-norm, 2e-3 of the output scale for ranking."""
import numpy as np
import pytest

import bm
import mlp_oracle as mo

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 511, 512, 640, 1025, 2100])
def test_gradients_across_split_sums(rows):
    rng = np.random.default_rng(rows)
    p = mo.init_params(rows).astype(np.float32)
    x = rng.normal(size=(rows, mo.IN)).astype(np.float32)
    t = rng.normal(size=rows).astype(np.float32)
    with bm.Mlp(seed=1) as net:
        net.set_params(p)
        loss, g = net.train_step(x, t, lr=0.0)
        y = net.forward(x)
    want_loss, want = mo.forward_backward(p, x, t, bf16_path=True)
    assert abs(loss - want_loss) <= 1e-3 * max(1.0, want_loss)
    for name, a, b in ((k, mo.unpack(g)[k], mo.unpack(want)[k]) for k, _ in mo.SIZES):
        assert np.linalg.norm(a - b) <= 2e-3 * np.linalg.norm(b) + 1e-7, name
    ref = mo.forward(p, x, bf16_path=True)
    assert np.abs(y - ref).max() <= 1e-3 * max(1.0, float(np.abs(ref).max()))


@pytest.mark.parametrize("k", [1, 128, 129, 148 * 128, 148 * 128 + 1, 2 * 148 * 128 + 77, 5 * 148 * 128 - 3])
def test_ranking_at_tile_edges(cfg0, k):
    rng = np.random.default_rng(k)
    a = rng.integers(1, cfg0["n"] + 1, k).astype(np.int32)
    b = rng.integers(1, cfg0["n"] + 1, k).astype(np.int32)
    with bm.Engine.from_pair(cfg0) as E, bm.Mlp(seed=5) as net:
        E.set_mapping(cfg0["map0"])
        y = net.rank_pairs(E, a, b)
        f1, f2 = net.features(E)
        at = np.unique(np.concatenate([np.arange(min(k, 200)), np.arange(max(0, k - 200), k), rng.integers(0, k, 500)]))
        x = mo.pair_inputs(f1, f2, cfg0["map0"], a[at] - 1, b[at] - 1)
        ref = mo.forward(net.get_params(), x, bf16_path=True)
    assert np.abs(y[at] - ref).max() <= 2e-3 * max(1.0, float(np.abs(ref).max()))
