"""The order of the profit rows is made with the first profit matrix, not with
every engine: an engine that only scores pays neither its time nor its memory."""
import numpy as np
import pytest

import bm
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,e", [(200, 3000), (1501, 30_000), (21_000, 60_000)])   # the last sorts by radix
def test_made_with_the_first_profit_matrix(n, e):
    g = bm.generate(bm.gen_params(n=n, e=e, seed=n))
    O = oracle.Oracle.from_pair(g)
    with bm.Engine.from_pair(g) as E:
        E.set_mapping(g["map0"])
        E.pair_deltas([1], [2])
        held = E.info()["device_bytes"]
        row = E.profit_row(1)
        made = E.info()["device_bytes"] - held
        # the matrix (rows of whole 16 bytes), its matching and inverse, the order
        assert made >= 4 * n * ((n + 3) // 4 * 4) + 8 * (n + 1) + 4 * n
        held = E.info()["device_bytes"]
        assert np.array_equal(E.profit_row(1), row) and E.info()["device_bytes"] == held
        m = g["map0"].copy()
        E.sweep()
        O.sweep(m)
        assert np.array_equal(E.get_mapping(), m)
