"""A batch of many small instances, of both entry widths: matchings set, scored and
read in one pass, each its own (instances lie along a launch's first dimension)."""
import numpy as np
import pytest

import bm
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, bm.BM_FLAG_FORCE_I32])
def test_many_small_instances(flags):
    rng = np.random.default_rng(4)
    pairs = []
    for i in range(300):
        n = int(rng.integers(2, 60)) if i % 50 else 1500   # one to six blocks of a matching
        e = int(rng.integers(0, 6 * n))
        s, d = rng.integers(1, n + 1, (2, e)).astype(np.int32)
        w = rng.integers(1, 50, e).astype(np.int32)
        pairs.append(dict(n=n, src1=s, dst1=d, w1=w, src2=d, dst2=s, w2=w[::-1].copy(),
                          map0=np.concatenate([[0], rng.permutation(n) + 1]).astype(np.int32)))
    with bm.Batch(pairs, flags) as B:
        B.set_mappings([g["map0"] for g in pairs])
        assert list(B.scores()) == [oracle.Oracle.from_pair(g).score(g["map0"]) for g in pairs]
        for m, g in zip(B.get_mappings(), pairs):
            assert np.array_equal(m, g["map0"])
        B.sweeps(2)
        got, scores = B.get_mappings(), B.scores()
    for g, m, sc in zip(pairs, got, scores):
        O, want = oracle.Oracle.from_pair(g), g["map0"].copy()
        O.sweep(want)
        O.sweep(want)
        assert np.array_equal(m, want) and O.score(m) == sc
