"""A batch of one instance sets and reads its matching by the instance's own
calls; two go through the batch's staging pass.  Same results, same errors."""
import numpy as np
import pytest

import bm
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2])
def test_set_and_get(count):
    pairs = [bm.generate(bm.gen_params(n=n, e=12 * n, seed=n)) for n in (301, 450)[:count]]
    with bm.Batch(pairs) as B:
        with pytest.raises(bm.BMError) as e:
            B.get_mappings()
        assert e.value.status == bm.BM_E_STATE and "instance 0" in str(e.value)
        maps = [g["map0"] for g in pairs]
        B.set_mappings(maps)
        for a, b in zip(B.get_mappings(), maps):
            assert np.array_equal(a, b)
        scores = [oracle.Oracle.from_pair(g).score(g["map0"]) for g in pairs]
        assert list(B.scores()) == scores
        bad = [m.copy() for m in maps]
        bad[0][1] = bad[0][2]                     # two vertices on one image
        with pytest.raises(bm.BMError) as e:
            B.set_mappings(bad)
        assert e.value.status == bm.BM_E_INPUT and "instance 0" in str(e.value)
        for a, b in zip(B.get_mappings(), maps):  # nothing was set
            assert np.array_equal(a, b)
        B.sweeps(2)
        got = B.get_mappings()
    for g, m in zip(pairs, got):
        O, want = oracle.Oracle.from_pair(g), g["map0"].copy()
        O.sweep(want)
        O.sweep(want)
        assert np.array_equal(m, want)
