"""Sizes around the profit matrix's row pitch and the combine's tiles: n mod 4
in 0..3, n at, below and above one and two tiles of 64 (32 in batches), with and
without the tensor-core hub terms.  All deltas, best partners (through the
sweep's candidates) and moves must equal the oracle's exactly."""
import numpy as np
import pytest

import bm
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 5, 31, 33, 63, 64, 65, 66, 67, 127, 128, 129, 257, 258, 259, 1003])
@pytest.mark.parametrize("flags", [0, bm.BM_FLAG_FORCE_I32, bm.BM_FLAG_NO_HUB_GEMM])
def test_deltas_and_sweeps(n, flags):
    g = bm.generate(bm.gen_params(n=n, e=min(n * (n - 1) // 2, 40 * n), seed=7 + n, wmax=90))
    O = oracle.Oracle.from_pair(g)
    m = g["map0"].copy()
    if n > 8:
        m[3] = m[n // 2] = 0   # unmatched vertices
    with bm.Engine.from_pair(g, flags) as E:
        E.set_mapping(m)
        np.testing.assert_array_equal(E.all_deltas(), O.all_deltas(m))
        for _ in range(2):
            st, ost = E.sweep(), O.sweep(m)
            for k in ("candidates", "committed", "best_delta"):
                assert st[k] == ost[k], k
            np.testing.assert_array_equal(E.get_mapping(), m)
        st, ost = E.sweep(incremental=True), O.sweep(m)
        assert st["committed"] == ost["committed"]
        E.lookup_descent(2)
        O.best_swap_descent(m, 2)
        np.testing.assert_array_equal(E.get_mapping(), m)


def test_batch_of_ragged_sizes():
    ns = (61, 64, 95, 129, 254, 383, 641)
    pairs = [bm.generate(bm.gen_params(n=n, e=15 * n, seed=n, wmax=90)) for n in ns]
    for schedule in ((True, 1024, 32), (True, 1024, 64), (False, 256, 32), (False, 512, 64)):
        with bm.Batch(pairs) as B:
            B.set_schedule(*schedule)
            B.set_mappings([g["map0"] for g in pairs])
            B.sweeps(2)
            got = B.get_mappings()
        for g, m in zip(pairs, got):
            want = g["map0"].copy()
            O = oracle.Oracle.from_pair(g)
            O.sweep(want)
            O.sweep(want)
            np.testing.assert_array_equal(m, want)
