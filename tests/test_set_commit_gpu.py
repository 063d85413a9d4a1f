"""The grid-wide set commit at the sizes where its windows can go wrong: fewer
candidates than a window, one more or less than a window, many windows; a
vertex that belongs to most candidates; dense pairs where every two candidates
are adjacent; re-verification budgets that end inside a window.  Moves and
counts must equal the oracle's one-at-a-time rule exactly."""
import numpy as np
import pytest

import bm
import oracle

pytestmark = pytest.mark.gpu

COUNTS = ("candidates", "scanned", "verified", "committed", "best_delta")


def _star(n, seed):
    """Two hubs joined to every vertex both ways, a sparse rest: the hubs are in most candidates."""
    rng = np.random.default_rng(seed)
    s, d = [], []
    for h in (1, 2):
        for v in range(3, n + 1):
            s += [h, v]
            d += [v, h]
    k = 2 * n
    s += list(rng.integers(3, n + 1, k))
    d += list(rng.integers(3, n + 1, k))
    s, d = np.array(s, np.int32), np.array(d, np.int32)
    keep = s != d
    s, d = s[keep], d[keep]
    perm = rng.permutation(n).astype(np.int32) + 1
    return dict(n=n, src1=s, dst1=d, w1=rng.integers(1, 40, len(s)).astype(np.int32), src2=perm[s - 1],
                dst2=perm[d - 1], w2=rng.integers(1, 40, len(s)).astype(np.int32),
                map0=np.concatenate([[0], rng.permutation(n) + 1]).astype(np.int32))


def _pair(shape, n, seed):
    if shape == "star":
        return _star(n, seed)
    e = n * (n - 1) // 3 if shape == "dense" else 6 * n
    return bm.generate(bm.gen_params(n=n, e=e, seed=seed, wmax=200))


@pytest.mark.parametrize("shape,n", [("dense", 5), ("dense", 140), ("dense", 400), ("sparse", 127), ("sparse", 1500),
                                     ("star", 130), ("star", 700)])
@pytest.mark.parametrize("flags", [0, bm.BM_FLAG_FORCE_I32])
def test_sweeps_match_oracle(shape, n, flags):
    g = _pair(shape, n, 17 + n)
    O = oracle.Oracle.from_pair(g)
    with bm.Engine.from_pair(g, flags) as E:
        for max_candidates, max_verify in ((0, -1), (0, 0), (0, 7), (1, -1), (127, -1), (128, 3), (129, -1)):
            m = g["map0"].copy()
            E.set_mapping(m)
            for _ in range(3):
                st, ost = E.sweep(max_candidates, max_verify), O.sweep(m, max_candidates, max_verify)
                assert {k: st[k] for k in COUNTS} == {k: ost[k] for k in COUNTS}
                np.testing.assert_array_equal(E.get_mapping(), m)
            assert E.score() == O.score(m)


@pytest.mark.parametrize("shape,n", [("dense", 40), ("dense", 300), ("sparse", 1500), ("star", 300)])
@pytest.mark.parametrize("flags,max_candidates,max_verify", [(0, 0, -1), (0, 129, 9), (bm.BM_FLAG_FORCE_I32, 0, 0)])
def test_rounds_match_oracle(shape, n, flags, max_candidates, max_verify):
    g = _pair(shape, n, 31 + n)
    O = oracle.Oracle.from_pair(g)
    m = g["map0"].copy()
    with bm.Engine.from_pair(g, flags) as E:
        E.set_mapping(m)
        for r in range(2):
            kw = dict(partners=24, seed=50 + r, max_candidates=max_candidates, max_verify=max_verify)
            for mine, want in ((E.triple_round, O.triple_round), (E.quad_round, O.quad_round)):
                st, ost = mine(**kw), want(m, **kw)
                assert {k: st[k] for k in COUNTS} == {k: ost[k] for k in COUNTS}
                np.testing.assert_array_equal(E.get_mapping(), m)
        assert E.score() == O.score(m)


@pytest.mark.parametrize("n", [2, 31, 33, 20480, 20481])
def test_candidate_sort_at_its_edges(n):
    """Below, at and above the largest size the counting sort takes, and fewer
    rows than one of its blocks; sparse pairs keep the oracle quick."""
    g = bm.generate(bm.gen_params(n=n, e=max(1, n // 2), seed=n, wmax=60))
    O = oracle.Oracle.from_pair(g)
    m = g["map0"].copy()
    with bm.Engine.from_pair(g) as E:
        E.set_mapping(m)
        st, ost = E.sweep(), O.sweep(m)
        assert {k: st[k] for k in COUNTS} == {k: ost[k] for k in COUNTS}
        np.testing.assert_array_equal(E.get_mapping(), m)
        assert E.score() == O.score(m)
