"""Best swaps of hubs, whose G2 lists are walked four entries per thread and
whose rows are summed in shared memory: list lengths around a warp's and a
block's step of entries, and around a quarter of the row.  The mapping after
every descent must equal the oracle's."""
import numpy as np
import pytest

import bm
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hub", [31, 33, 127, 129, 511, 600])
@pytest.mark.parametrize("flags", [0, bm.BM_FLAG_FORCE_I32])
def test_swaps_of_hubs(hub, flags):
    n = 620
    rng = np.random.default_rng(hub)
    g = bm.generate(bm.gen_params(n=n, e=4 * n, seed=hub, wmax=9))
    for s in "12":   # a vertex with `hub` out-edges and one with `hub` in-edges on both sides
        ids = rng.permutation(np.arange(3, n + 1))[:hub].astype(np.int32)
        ones = np.ones(hub, np.int32)
        w = rng.integers(1, 9, 2 * hub).astype(np.int32)
        g["src" + s] = np.concatenate([g["src" + s], ones, ids])
        g["dst" + s] = np.concatenate([g["dst" + s], ids, 2 * ones])
        g["w" + s] = np.concatenate([g["w" + s], w])
    m = g["map0"].copy()
    m[5] = 0
    O = oracle.Oracle.from_pair(g)
    with bm.Engine.from_pair(g, flags) as E:
        E.set_mapping(m)
        E.lookup_descent(8)
        O.best_swap_descent(m, 8)
        np.testing.assert_array_equal(E.get_mapping(), m)
        assert E.score() == O.score(m)
