"""Engines of different sizes used by several host threads at once.

A kernel's dynamic shared memory limit belongs to the process.  Two threads that
set it to their own engine's need before each launch get in each other's way:
the smaller engine's setting between the larger one's setting and launch makes
that launch fail."""
import threading

import numpy as np
import pytest

import bm

pytestmark = pytest.mark.gpu


def _together(jobs, rounds):
    """Each job repeatedly in a thread of its own; every result is the first one's."""
    want = [job() for job in jobs]
    bad = []
    go = threading.Barrier(len(jobs))

    def work(i):
        go.wait()
        try:
            for _ in range(rounds):
                if not np.array_equal(jobs[i](), want[i]):
                    bad.append((i, "another result"))
                    return
        except bm.BMError as e:
            bad.append((i, str(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(jobs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad


@pytest.mark.parametrize("call", ["sweep", "triple", "quad", "update", "first"])
def test_engines_of_three_sizes(call):
    engines = []
    for n, d in ((300, 12), (700, 12), (4000, 6)):
        g = bm.generate(bm.gen_params(n=n, e=n * d, seed=n))
        engines.append((bm.Engine.from_pair(g), g["map0"]))

    def job(E, m):
        E.set_mapping(m)
        if call == "sweep":
            E.sweep()
        elif call == "update":
            E.sweep(incremental=True)
            E.sweep(incremental=True)
            E.lookup_descent(3)
        elif call == "triple":
            E.triple_round(partners=8, seed=1)
        elif call == "quad":
            E.quad_round(partners=4, seed=1)
        else:
            E.first_improvement(1)
        return E.get_mapping()

    if call == "first":
        engines = engines[:2]
    try:
        _together([lambda E=E, m=m: job(E, m) for E, m in engines], 15 if call == "first" else 150)
    finally:
        for E, _ in engines:
            E.close()


def test_greedy_of_three_sizes():
    graphs = [bm.generate(bm.gen_params(n=n, e=n * 8, seed=n)) for n in (100, 250, 400)]
    _together([lambda g=g: bm.greedy_match(g)[0] for g in graphs], 40)
