"""The greedy matching where a slice of the cluster has as many candidates as a
CTA has threads (n = 16 x 512), one more, and around the line above it from
which the grid takes over (2 E1 E2 / n = 1e7): identical to the oracle."""
import numpy as np
import pytest

import bm
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,e", [(8192, 25_000), (8193, 25_000), (8300, 200_000), (8300, 208_000)])
def test_matches_oracle(n, e):
    g = bm.generate(bm.gen_params(n=n, e=e, seed=n + e, wmax=50))
    assert np.array_equal(bm.greedy_match(g)[0], oracle.greedy_match(g))
