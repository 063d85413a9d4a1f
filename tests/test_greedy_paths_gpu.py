"""The greedy matching on both sides of its dispatch and at the edges of the
cluster's slices (n below, at and above its 16 CTAs and their multiples), with
hub vertices whose edges take several chunks: identical to the oracle."""
import numpy as np
import pytest

import bm
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,e", [(2, 2), (15, 60), (16, 60), (17, 60), (33, 300), (511, 5000), (1200, 24000),
                                 (1000, 153000),   # 2 E1 E2 / n = 4.7e7: the cluster
                                 (1000, 157000)])  # 4.9e7: the grid
def test_matches_oracle(n, e):
    g = bm.generate(bm.gen_params(n=n, e=min(e, n * (n - 1) // 2 if n < 20 else e), seed=n + e, wmax=50))
    assert np.array_equal(bm.greedy_match(g)[0], oracle.greedy_match(g))


def test_hub_rows_take_several_chunks():
    n = 1500
    rng = np.random.default_rng(8)
    s = np.concatenate([np.full(n - 1, 1), np.arange(2, n + 1), rng.integers(1, n + 1, 4 * n)]).astype(np.int32)
    d = np.concatenate([np.arange(2, n + 1), np.full(n - 1, 1), rng.integers(1, n + 1, 4 * n)]).astype(np.int32)
    w = rng.integers(0, 30, len(s)).astype(np.int32)
    perm = rng.permutation(n).astype(np.int32) + 1
    g = dict(n=n, src1=s, dst1=d, w1=w, src2=perm[s - 1], dst2=perm[d - 1], w2=rng.integers(1, 30, len(s)).astype(np.int32))
    assert np.array_equal(bm.greedy_match(g)[0], oracle.greedy_match(g))
