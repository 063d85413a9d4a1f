"""Row bests of sparse batch instances without the profit matrix: sizes around
the lines of its row accumulators, lists of every length class (up to 64
entries, up to 4,096, longer), self-loops, unmatched vertices, equal deltas, and
32-bit entries.  Every instance must end where it ends alone."""
import numpy as np
import pytest

import bm

pytestmark = pytest.mark.gpu


def _pair(n, degree, seed, hub=0, loops=0, unmatched=0, wmax=4):
    rng = np.random.default_rng(seed)

    def side():
        e = degree * n
        src, dst = rng.integers(1, n + 1, e), rng.integers(1, n + 1, e)
        if hub:   # one vertex with `hub` out-edges, another with `hub` in-edges
            ids = rng.permutation(n)[:hub] + 1
            src = np.concatenate([src, np.full(hub, 1 + n // 3), ids])
            dst = np.concatenate([dst, ids, np.full(hub, 1 + n // 2)])
        keep = src != dst
        src, dst = src[keep], dst[keep]
        own = rng.permutation(n)[:loops] + 1
        src, dst = np.concatenate([src, own]), np.concatenate([dst, own])
        pair = np.unique(src.astype(np.int64) * (n + 1) + dst)
        src, dst = (pair // (n + 1)).astype(np.int32), (pair % (n + 1)).astype(np.int32)
        return src, dst, rng.integers(1, wmax + 1, len(src)).astype(np.int32)

    g = dict(n=n)
    for s in "12":
        g["src" + s], g["dst" + s], g["w" + s] = side()
    m = np.zeros(n + 1, np.int32)
    m[1:] = rng.permutation(n) + 1
    m[1 + rng.permutation(n)[:unmatched]] = 0
    g["map0"] = m
    return g


SETS = {
    "small": [_pair(n, 3, n, loops=n // 4, unmatched=n // 5) for n in (2, 3, 31, 32, 33, 127, 130, 257)],
    "lists": [_pair(1500, 6, 1, hub=64), _pair(1501, 6, 2, hub=65), _pair(1502, 6, 3, hub=700, loops=300),
              _pair(5003, 4, 4, hub=4600, unmatched=900)],
    "accumulators": [_pair(n, 8, n, unmatched=n // 50) for n in (6500, 6600, 6700, 6911, 8189, 8192)],
    "dense": [_pair(200, 60, 5), _pair(900, 10, 6, loops=20), _pair(90, 40, 7)],
}


@pytest.mark.parametrize("name", sorted(SETS))
@pytest.mark.parametrize("flags", [0, bm.BM_FLAG_FORCE_I32])
def test_instances_end_where_they_end_alone(name, flags):
    pairs = SETS[name]
    with bm.Batch(pairs, flags) as B:
        B.set_schedule(True, 1024, 64)
        B.set_mappings([g["map0"] for g in pairs])
        committed, _ = B.sweeps(3)
        got = B.get_mappings()
    for g, m, c in zip(pairs, got, committed):
        with bm.Engine.from_pair(g, bm.BM_FLAG_NO_HUB_GEMM | flags) as E:
            E.set_mapping(g["map0"])
            want = sum(E.sweep()["committed"] for _ in range(3))
            assert c == want, g["n"]
            np.testing.assert_array_equal(m, E.get_mapping())


def test_a_bad_matching_stops_at_its_instance():
    pairs = [_pair(n, 4, n, unmatched=2) for n in (40, 70, 55)]
    first = [g["map0"] for g in pairs]
    with bm.Batch(pairs) as B:
        with pytest.raises(bm.BMError):
            B.get_mappings()
        B.set_mappings(first)
        scores = B.scores()
        other = [np.concatenate([m[:1], np.roll(m[1:], 3)]) for m in first]
        other[1] = other[1].copy()
        other[1][1] = other[1][2] = 7
        with pytest.raises(bm.BMError, match="instance 1: .*matched twice"):
            B.set_mappings(other)
        for want, m in zip((other[0], first[1], first[2]), B.get_mappings()):
            np.testing.assert_array_equal(m, want)
        assert (B.scores()[1:] == scores[1:]).all()
