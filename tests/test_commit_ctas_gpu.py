"""bm_sweep_opts.commit_ctas: the fewest CTAs of the set commit.  More of them
than the lists need, up to the whole GPU, make the same moves, and asking for
few is not slower than not asking."""
import numpy as np
import pytest

import bm
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,e", [(60, 400), (700, 4000)])   # short lists: 8 CTAs unless asked for more
def test_any_number_makes_the_same_moves(n, e):
    g = bm.generate(bm.gen_params(n=n, e=e, seed=n))
    O = oracle.Oracle.from_pair(g)
    for max_verify in (-1, 5):
        m = g["map0"].copy()
        want = [O.sweep(m, max_verify=max_verify)["committed"] for _ in range(3)]
        for ctas in (-1, 0, 1, 8, 9, 37, 148, 10_000):
            with bm.Engine.from_pair(g) as E:
                E.set_mapping(g["map0"])
                assert [E.sweep(max_verify=max_verify, commit_ctas=ctas)["committed"] for _ in range(3)] == want
                assert np.array_equal(E.get_mapping(), m), (max_verify, ctas)


def test_asking_for_few_is_not_slower():
    g = bm.generate(bm.gen_params(n=6000, e=600_000, seed=2))
    with bm.Engine.from_pair(g) as E:
        def best(ctas):
            ms = []
            for _ in range(8):
                E.set_mapping(g["map0"])
                ms.append(E.sweep(commit_ctas=ctas)["ms_commit"])
            return min(ms)
        best(0)
        assert best(1) <= 1.5 * best(0)   # one CTA alone takes seven times as long
