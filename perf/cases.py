"""Performance cases: the work a user has this engine do, through its public binding.

`listed()` names the cases, `draw(rng)` gives one more of the same ranges,
`prepare(case, seed)` makes what a user's program holds before the call (graph
pairs, an engine, a matching), `run(state)` is one pass through the public
entry points, `work(case)` counts the bytes and operations a pass cannot do
without, and `exact(case, seed)` is the 64-bit value of floating outputs.

Graph pairs come from the engine's own generator, in the shapes of the
repository's workloads: power-law out-degrees, geometric weights with an
optional heavy tail, G2 a relabelled and perturbed G1.  Every pass starts by
setting a matching from host memory and ends with the results on the host, as
the command-line tools do.  All results but the network's are whole numbers.
"""
import math
import os
import sys

import numpy as np

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "brain-match_b200"))
import bm  # noqa: E402

MLP_IN, MLP_HID = 128, 256


def listed():
    return [
        # one pairwise sweep of a small pair (the repository's N=1,000 workload): a call of many short launches
        dict(name="sweep_n1000", kind="sweep", n=1000, e=20_000, tail=0.0, i32=False, warm=0),
        # the same call on a mid-sized pair of odd size whose weights need 32-bit entries
        dict(name="sweep_n6007_i32", kind="sweep", n=6007, e=300_000, tail=1e-3, i32=True, warm=2),
        # the headline: a sweep at connectome size, four sweeps into a descent from a random matching
        dict(name="sweep_n18524", kind="sweep", n=18524, e=5_000_000, tail=1e-3, i32=False, warm=4),
        # a whole hill climb to a local optimum, odd size: rebuilds first, then updates of the profit matrix
        dict(name="descent_n7001", kind="descent", n=7001, e=700_000, tail=1e-3, i32=False),
        # the reference's sequential first-improvement order to its fixed point
        dict(name="first_n600", kind="first", n=600, e=12_000, tail=0.0, i32=False),
        # the `triple` tool's work on a swept matching: a 3-cycle round, then a 4-set round
        dict(name="rounds_n8192", kind="rounds", n=8192, e=1_000_000, tail=1e-3, i32=False, warm=8, triples=256,
             quads=64),
        # many independent pairs of uneven size swept together (the repository's batch workload)
        dict(name="batch_64", kind="batch", count=64, nmin=500, nmax=8000, degree=20, sweeps=3),
        # exact best-swap descent: 64 swaps on the exact table
        dict(name="lookup_n8192", kind="lookup", n=8192, e=1_000_000, tail=1e-3, i32=False, swaps=64),
        # all pair deltas to the host, then the deltas of a list of pairs (odd size)
        dict(name="deltas_n3001", kind="deltas", n=3001, e=120_000, tail=0.0, i32=False, pairs=20_000),
        # one forward and backward pass of the proposal network with its update, the engine's batch of 1,024 rows
        dict(name="train_step_1024", kind="train", rows=1024),
        # a learned sweep: rank a pool of candidate swaps, evaluate the best exactly, commit
        dict(name="learned_n8192", kind="learned", n=8192, e=1_000_000, tail=1e-3, i32=False, pool=64),
        # the greedy initial matching from edge lists
        dict(name="greedy_n3000", kind="greedy", n=3000, e=150_000, tail=0.0),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pair(rng, nlo, nhi, dlo, dhi, i32=True):
    n = _logint(rng, nlo, nhi)
    e = min(int(n * math.exp(rng.uniform(math.log(dlo), math.log(dhi)))), n * (n - 1) // 4)
    return dict(n=n, e=e, tail=rng.choice([0.0, 1e-3]), i32=i32 and rng.random() < 0.25)


def draw(rng):
    kind = rng.choice(["sweep", "sweep", "descent", "first", "rounds", "batch", "lookup", "deltas", "train", "learned",
                       "greedy"])
    if kind == "sweep":
        return dict(_pair(rng, 500, 18_524, 15, 270), kind=kind, warm=rng.randint(0, 6))
    if kind == "descent":
        return dict(_pair(rng, 1000, 8000, 20, 120), kind=kind)
    if kind == "first":
        return dict(_pair(rng, 200, 700, 10, 25), kind=kind)
    if kind == "rounds":
        return dict(_pair(rng, 1500, 10_000, 20, 140), kind=kind, warm=rng.randint(2, 8),
                    triples=rng.choice([64, 128, 256]), quads=rng.choice([16, 32, 64]))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(8, 64), nmin=rng.randint(200, 1000), nmax=rng.randint(1500, 8000),
                    degree=rng.randint(12, 24), sweeps=rng.randint(1, 3))
    if kind == "lookup":
        return dict(_pair(rng, 1000, 10_000, 20, 140), kind=kind, swaps=rng.randint(16, 96))
    if kind == "deltas":
        return dict(_pair(rng, 500, 4000, 15, 60), kind=kind, pairs=_logint(rng, 1000, 40_000))
    if kind == "train":
        return dict(kind=kind, rows=_logint(rng, 200, 8000))
    if kind == "learned":
        return dict(_pair(rng, 1500, 10_000, 20, 140), kind=kind, pool=rng.choice([32, 64, 100]))
    n = _logint(rng, 800, 4000)
    return dict(kind=kind, n=n, e=n * rng.randint(15, 60), tail=0.0)


def _generate(case, seed):
    return bm.generate(bm.gen_params(n=case["n"], e=case["e"], seed=0x5EED0000 + 7919 * seed,
                                     wmax=30_000 if case["tail"] else 5000, tail_prob=case["tail"]))


def _train_inputs(case, seed):
    """Network parameters, rows and targets as training meets them: z-scored features, sign(d) log1p|d|."""
    rng = np.random.default_rng([seed, case["rows"]])
    k1, k2 = math.sqrt(6 / MLP_IN), math.sqrt(6 / MLP_HID)
    params = np.concatenate([rng.uniform(-k1, k1, MLP_HID * MLP_IN), rng.normal(0, 0.05, MLP_HID),
                             rng.uniform(-k2, k2, MLP_HID * MLP_HID), rng.normal(0, 0.05, MLP_HID),
                             rng.uniform(-k2, k2, MLP_HID), [0.1]]).astype(np.float32)
    x = rng.normal(size=(case["rows"], MLP_IN)).astype(np.float32)
    d = np.round(rng.normal(0, 30, case["rows"]))
    return params, x, (np.sign(d) * np.log1p(np.abs(d))).astype(np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        params, x, t = _train_inputs(case, seed)
        net = bm.Mlp(seed=1)
        net.set_params(params)
        return dict(kind=kind, net=net, x=x, t=t)
    if kind == "batch":
        rng = np.random.default_rng(case["count"])  # the sizes belong to the case, the pairs to the seed
        ns = np.exp(rng.uniform(np.log(case["nmin"]), np.log(case["nmax"]), case["count"])).astype(int)
        pairs = [bm.generate(bm.gen_params(n=int(n), e=case["degree"] * int(n), seed=0xBA7C0000 + 7919 * seed + i))
                 for i, n in enumerate(ns)]
        batch = bm.Batch(pairs)
        maps = [g["map0"] for g in pairs]
        batch.set_mappings(maps)
        batch.autotune()
        return dict(kind=kind, batch=batch, maps=maps, sweeps=case["sweeps"])
    g = _generate(case, seed)
    if kind == "greedy":
        return dict(kind=kind, g=g)
    s = dict(kind=kind, case=case, start=g["map0"],
             engine=bm.Engine.from_pair(g, bm.BM_FLAG_FORCE_I32 if case["i32"] else 0))
    if case.get("warm"):  # the matching a descent has reached
        s["engine"].set_mapping(g["map0"])
        for _ in range(case["warm"]):
            s["engine"].sweep()
        s["start"] = s["engine"].get_mapping()
    if kind == "deltas":
        rng = np.random.default_rng([seed, case["pairs"]])
        m1 = rng.integers(1, case["n"] + 1, case["pairs"])
        m2 = (m1 + rng.integers(0, case["n"] - 1, case["pairs"])) % case["n"] + 1
        s["m1"], s["m2"] = m1.astype(np.int32), m2.astype(np.int32)
    if kind == "learned":
        s["net"], s["seed"] = bm.Mlp(seed=seed), seed
    return s


def run(s):
    kind = s["kind"]
    if kind == "train":
        loss, grads = s["net"].train_step(s["x"], s["t"], lr=1e-3)
        return dict(loss=np.float32(loss), grads=grads)
    if kind == "batch":
        s["batch"].set_mappings(s["maps"])
        committed, _ = s["batch"].sweeps(s["sweeps"])
        return dict(maps=np.concatenate(s["batch"].get_mappings()), committed=committed)
    if kind == "greedy":
        return bm.greedy_match(s["g"])[0]
    eng, case = s["engine"], s["case"]
    eng.set_mapping(s["start"])
    if kind == "deltas":
        return dict(all=eng.all_deltas(), pairs=eng.pair_deltas(s["m1"], s["m2"]))
    if kind == "sweep":
        st = eng.sweep()
        counts = [st[k] for k in ("candidates", "scanned", "verified", "committed", "best_delta")]
    elif kind == "descent":
        sweeps, committed, last = 0, 0, 1
        while last:
            st = eng.sweep(incremental=True)
            last = st["committed"]
            sweeps, committed = sweeps + 1, committed + last
        counts = [sweeps, committed]
    elif kind == "first":
        counts = list(eng.first_improvement(100))
    elif kind == "rounds":
        t = eng.triple_round(partners=case["triples"], seed=11, incremental=True)
        st = eng.quad_round(partners=case["quads"], seed=12, incremental=True)
        counts = [r[k] for r in (t, st) for k in ("candidates", "scanned", "verified", "committed", "best_delta")]
        counts += [t["triples"], st["quads"]]
    elif kind == "lookup":
        st = eng.lookup_descent(case["swaps"])
        counts = [st["swaps"], st["converged"]]
    else:
        st = s["net"].learned_sweep(eng, pool=case["pool"], top_fraction=0.02, seed=s["seed"])
        counts = [st[k] for k in ("scanned", "verified", "committed")]
    return dict(map=eng.get_mapping(), counts=np.array(counts, np.int64),
                score=eng.score() if kind == "first" else st["score_after"])


def _terms(n, e):
    """Nonzero min terms of the profit matrix at a random matching, one min and one add each."""
    return 2 * 2.0 * e * e / n


def work(case):
    kind = case["kind"]
    if kind == "train":
        rows = case["rows"]
        params = MLP_HID * (MLP_IN + MLP_HID + 3) + 1
        fwd = 2.0 * rows * MLP_HID * (MLP_IN + MLP_HID + 1)
        return dict(bytes=4.0 * (rows * (MLP_IN + 1) + 3 * params), flops=fwd * 2 + 2.0 * rows * MLP_HID * MLP_HID)
    if kind == "batch":
        lo, hi = case["nmin"], case["nmax"]
        mean = (hi - lo) / math.log(hi / lo)
        mean2 = (hi * hi - lo * lo) / (2 * math.log(hi / lo))
        per = 2 * 2.0 * case["degree"] ** 2 * mean + 1.5 * mean2
        return dict(bytes=case["count"] * mean * (8.0 * case["degree"] + 8), flops=case["count"] * case["sweeps"] * per)
    n, e = case["n"], case["e"]
    if kind == "greedy":  # every matched edge's G2 list once; a score per vertex pair
        return dict(bytes=24.0 * e + 4 * n, flops=_terms(n, e) + 6.0 * n * n)
    entry = 8 if case["i32"] else 4
    lists, maps = 2.0 * e * entry, 8.0 * n
    combine = 1.5 * n * n
    if kind == "sweep":
        return dict(bytes=lists + maps, flops=_terms(n, e) + combine)
    if kind == "descent":  # the profit matrix once, then a combine per sweep of about 40
        return dict(bytes=lists + maps, flops=_terms(n, e) + 40 * combine)
    if kind == "first":  # about five passes, each edge of both vertices per pair
        return dict(bytes=lists + maps, flops=5 * n * 8.0 * e)
    if kind == "rounds":
        return dict(bytes=lists + maps, flops=_terms(n, e) + n * (case["triples"] * 2 * 10.0 + case["quads"] * 23 * 10.0))
    if kind == "lookup":  # the table once, then the changes of each swap
        return dict(bytes=lists + maps, flops=_terms(n, e) + case["swaps"] * 8.0 * (e / n) ** 2)
    if kind == "deltas":
        return dict(bytes=lists + maps + 2.0 * n * (n - 1) + 12.0 * case["pairs"],
                    flops=_terms(n, e) + combine + case["pairs"] * 8.0 * e / n)
    return dict(bytes=lists + maps, flops=2.0 * n * case["pool"] * MLP_HID * MLP_HID + 2.0 * n * 2 * MLP_HID * MLP_IN)


def exact(case, seed):
    if case["kind"] != "train":  # whole numbers
        return None
    params, x, t = (v.astype(np.float64) for v in _train_inputs(case, seed))
    at = np.cumsum([0, MLP_HID * MLP_IN, MLP_HID, MLP_HID * MLP_HID, MLP_HID, MLP_HID, 1])
    w1, b1, w2, b2, w3, b3 = (params[i:j] for i, j in zip(at[:-1], at[1:]))
    w1, w2 = w1.reshape(MLP_HID, MLP_IN), w2.reshape(MLP_HID, MLP_HID)
    h1 = np.maximum(x @ w1.T + b1, 0)
    h2 = np.maximum(h1 @ w2.T + b2, 0)
    r = h2 @ w3 + b3 - t
    dy = 2 * r / len(x)
    d2 = np.where(h2 > 0, dy[:, None] * w3, 0)
    d1 = np.where(h1 > 0, d2 @ w2, 0)
    grads = np.concatenate([(d1.T @ x).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), h2.T @ dy, [dy.sum()]])
    return dict(loss=np.float64(np.mean(r * r)), grads=grads)
