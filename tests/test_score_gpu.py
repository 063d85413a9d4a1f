"""The score at the edges of its entry runs and of its 33-way row search: sizes
around 33 and 33^2 rows, edge counts around whole runs, empty rows before,
between and behind the others, self-loops and no edges at all."""
import numpy as np
import pytest

import bm
import oracle

pytestmark = pytest.mark.gpu


def _check(n, s, d, w, rng):
    t = rng.permutation(n) + 1
    m = np.concatenate([[0], t]).astype(np.int32)
    s2, d2, w2 = t[s - 1].astype(np.int32), t[d - 1].astype(np.int32), w[::-1].copy()
    g = dict(n=n, src1=s, dst1=d, w1=w, src2=s2, dst2=d2, w2=w2)
    O = oracle.Oracle.from_pair(g)
    with bm.Engine.from_pair(g) as E:
        E.set_mapping(m)
        assert E.score() == O.score(m)
        m[[1, n]] = m[[n, 1]]
        E.set_mapping(m)
        assert E.score() == O.score(m)


@pytest.mark.parametrize("n", [2, 3, 32, 33, 34, 35, 65, 1088, 1089, 1090, 1123, 5000])
@pytest.mark.parametrize("e", [0, 1, 31, 32, 33, 255, 256, 257, 4097])
def test_runs_and_rows(n, e):
    rng = np.random.default_rng(n * 10_007 + e)
    s, d = rng.integers(1, n + 1, (2, e)).astype(np.int32)
    _check(n, s, d, rng.integers(1, 100, e).astype(np.int32), rng)


@pytest.mark.parametrize("rows", [(1,), (700,), (1, 700), (350, 351)])
def test_all_edges_in_few_rows(rows):
    rng = np.random.default_rng(sum(rows))
    e = 3000
    s = rng.choice(rows, e).astype(np.int32)
    d = rng.integers(1, 701, e).astype(np.int32)
    _check(700, s, d, rng.integers(1, 100, e).astype(np.int32), rng)
