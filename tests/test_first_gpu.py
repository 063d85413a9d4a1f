"""The persistent first-improvement scans at their edges: fewer rows than CTAs,
passes that end inside a step, more steps than one launch takes, partial
matchings, self-loops, lists too long for a row per CTA (a warp per pair on
the whole grid), and a size whose rows do not fit shared memory; commits, passes, matching and score must equal
the oracle's sequential order exactly."""
import numpy as np
import pytest

import bm
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,e", [(2, 2), (3, 4), (33, 200), (150, 9000), (257, 2500), (420, 9000), (300, 15000)])
@pytest.mark.parametrize("flags", [0, bm.BM_FLAG_FORCE_I32])
def test_order_matches_oracle(n, e, flags):
    g = bm.generate(bm.gen_params(n=n, e=e, seed=n, wmax=300))
    rng = np.random.default_rng(n)
    loops = rng.integers(1, n + 1, max(1, n // 20)).astype(np.int32)   # G1 self-loops
    g["src1"], g["dst1"] = np.append(g["src1"], loops), np.append(g["dst1"], loops)
    g["w1"] = np.append(g["w1"], rng.integers(1, 9, len(loops)).astype(np.int32))
    O = oracle.Oracle.from_pair(g)
    with bm.Engine.from_pair(g, flags) as E:
        for passes, holes in ((0, 0), (1, 0), (2, n // 5), (1000, 0)):
            m = g["map0"].copy()
            m[rng.choice(np.arange(1, n + 1), holes, replace=False)] = 0
            E.set_mapping(m)
            got = E.first_improvement(passes)
            c, p, _ = O.first_improvement(m, passes)
            assert got == (c, p)
            np.testing.assert_array_equal(E.get_mapping(), m)
            assert E.score() == O.score(m)


def test_order_matches_oracle_beyond_shared_memory():
    n = 19600
    rng = np.random.default_rng(5)
    hot = rng.choice(np.arange(1, n + 1), 300, replace=False).astype(np.int32)   # the vertices with edges
    def edges(k):
        s, d = rng.choice(hot, k), rng.choice(hot, k)
        return s[s != d], d[s != d], rng.integers(1, 9, int((s != d).sum())).astype(np.int32)
    (s1, d1, w1), (s2, d2, w2) = edges(1500), edges(1500)
    g = dict(n=n, src1=s1, dst1=d1, w1=w1, src2=s2, dst2=d2, w2=w2)
    O = oracle.Oracle.from_pair(g)
    m = np.concatenate([[0], rng.permutation(n) + 1]).astype(np.int32)
    with bm.Engine.from_pair(g) as E:
        E.set_mapping(m)
        got = E.first_improvement(1)
        c, p, _ = O.first_improvement(m, 1)
        assert got == (c, p) and c > 0
        np.testing.assert_array_equal(E.get_mapping(), m)
        assert E.score() == O.score(m)
