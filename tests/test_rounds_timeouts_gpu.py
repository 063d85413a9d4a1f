"""The bounded waits of the 3-cycle and 4-set rounds' commit and of the
first-improvement exchange (one cluster, and the whole grid), made to run out by
bm_test_stall: BM_E_TIMEOUT, a matching is asked for, and the same call then
makes the moves it makes on an engine that never stalled."""
import numpy as np
import pytest

import bm

pytestmark = pytest.mark.gpu


def _runs_out(g, site, text, call):
    with bm.Engine.from_pair(g) as E:
        E.set_mapping(g["map0"])
        E.sweep()
        start = E.get_mapping()
        want = call(E)
        moved, score = E.get_mapping(), E.score()
    with bm.Engine.from_pair(g) as E:
        E.set_mapping(start)
        bm.test_stall(site)
        with pytest.raises(bm.BMError) as e:
            call(E)
        assert e.value.status == bm.BM_E_TIMEOUT
        assert text in str(e.value) and "timed out" in str(e.value)
        with pytest.raises(bm.BMError) as e:
            call(E)
        assert e.value.status == bm.BM_E_STATE
        E.set_mapping(start)
        got = call(E)
        assert np.array_equal(E.get_mapping(), moved) and E.score() == score
    return want, got


@pytest.mark.parametrize("incremental", [False, True])
def test_triple_round(cfg0, incremental):
    want, got = _runs_out(cfg0, bm.BM_STALL_COMMIT, "bm_triple_round: set commit wait",
                          lambda E: E.triple_round(partners=32, seed=1, incremental=incremental))
    assert want["committed"] == got["committed"] > 0


@pytest.mark.parametrize("incremental", [False, True])
def test_quad_round(cfg0, incremental):
    want, got = _runs_out(cfg0, bm.BM_STALL_COMMIT, "bm_quad_round: set commit wait",
                          lambda E: E.quad_round(partners=16, seed=1, incremental=incremental))
    assert want["committed"] == got["committed"] > 0


@pytest.mark.parametrize("n,e", [(300, 6000), (900, 60_000)])   # terms of a row: one cluster, the whole grid
def test_first_improvement(n, e):
    assert (4.0 * e / n * e / n <= 4096) == (n == 300)
    want, got = _runs_out(bm.generate(bm.gen_params(n=n, e=e, seed=12)), bm.BM_STALL_FIRST,
                          "bm_first_improvement: exchange wait", lambda E: E.first_improvement(1))
    assert want == got and got[0] > 0
