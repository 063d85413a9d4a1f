"""Timeouts inside a learned sweep: the ranking's tensor-core wait and the set
commit's exchange, made to run out by bm_test_stall (one wait that nothing
completes, with a short limit).  The call returns BM_E_TIMEOUT, the engine wants
a matching before anything else, and then works as if nothing had happened."""
import numpy as np
import pytest

import bm
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("site,text,pool", [(bm.BM_STALL_RANK, "tensor-core GEMM wait", 4),
                                            (bm.BM_STALL_RANK, "tensor-core GEMM wait", 128),
                                            (bm.BM_STALL_COMMIT, "set commit wait", 64)])
def test_learned_sweep_wait_runs_out(cfg0, site, text, pool):
    g = cfg0
    O = oracle.Oracle.from_pair(g)
    with bm.Engine.from_pair(g) as E, bm.Mlp(seed=7) as net:
        E.set_mapping(g["map0"])
        want = net.learned_sweep(E, pool=pool, seed=5)
        moved = E.get_mapping()
        E.set_mapping(g["map0"])
        E.sweep(incremental=True)                 # a kept profit matrix
        bm.test_stall(site)
        with pytest.raises(bm.BMError) as e:
            net.learned_sweep(E, pool=pool, seed=5)
        assert e.value.status == bm.BM_E_TIMEOUT and text in str(e.value) and "timed out" in str(e.value)
        for call in (E.sweep, lambda: net.learned_sweep(E), E.get_mapping):
            with pytest.raises(bm.BMError) as e:
                call()
            assert e.value.status == bm.BM_E_STATE
        E.set_mapping(g["map0"])
        assert E.score() == O.score(g["map0"])
        st = net.learned_sweep(E, pool=pool, seed=5)
        assert st["committed"] == want["committed"] and np.array_equal(E.get_mapping(), moved)
        assert E.score() == O.score(moved) == st["score_after"]
        m = moved.copy()
        E.sweep(incremental=True)
        O.sweep(m)
        assert np.array_equal(E.get_mapping(), m)


def test_ranking_wait_runs_out(cfg0):
    rng = np.random.default_rng(3)
    a, b = rng.integers(1, cfg0["n"] + 1, (2, 100_000)).astype(np.int32)
    with bm.Engine.from_pair(cfg0) as E, bm.Mlp(seed=7) as net:
        E.set_mapping(cfg0["map0"])
        y = net.rank_pairs(E, a, b)
        bm.test_stall(bm.BM_STALL_RANK)
        with pytest.raises(bm.BMError) as e:
            net.rank_pairs(E, a, b)
        assert e.value.status == bm.BM_E_TIMEOUT
        assert np.array_equal(net.rank_pairs(E, a, b), y)   # nothing was moved: the engine is usable at once
