"""The work that users of the engine have it do, as cases that can be timed.

Every case goes through the public Python API (Problem, Solver, Batch, Server)
and returns whole results: tours, costs and statistics of searches, candidates
and applied moves of neighbourhood passes, the constructed start tours.  All
results are whole numbers and have to stay equal bit for bit.

Instances are the benchmark's: integer coordinates in [0, 1000]^2, uniform or
eight Gaussian clusters with sigma 50, EUC_2D distances, depot 0 and seeded
random starts.  The sizes of a case are fixed by the case; coordinates, starts
and seeds of the constructor come from the seed.
"""
import os
import sys

import numpy as np

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "wamca-gpu-mi_gb300"))
import mlpgpu  # noqa: E402
from mlpgpu import workloads  # noqa: E402

ALL = mlpgpu.NB_ALL
UNCAPPED = 1 << 20


def _dvnd(name, n, wide=False, mask=ALL, iters=UNCAPPED, layout="uniform", rounded=True):
    return {"name": name, "kind": "dvnd", "n": n, "wide": wide, "mask": mask, "iters": iters, "layout": layout,
            "rounded": rounded}


def _batch(name, instances, starts, lo, hi, layout="clustered"):
    return {"name": name, "kind": "batch", "instances": instances, "starts": starts, "lo": lo, "hi": hi,
            "layout": layout}


def listed():
    return [
        # One search of a TSPLIB-sized small instance (berlin52's size): launches and latency.
        _dvnd("search_52", 52),
        # A small odd size with the reference's truncating distances, clustered.
        _dvnd("search_149", 149, layout="clustered", rounded=False),
        # One mid-size search, as a caller of a DVND step inside an ILS makes it.
        _dvnd("search_417", 417),
        # The benchmark's headline: one n = 1000 search to its local optimum.
        _dvnd("search_1000", 1000),
        # The same size with exact 64-bit latencies.
        _dvnd("search_1000_wide", 1000, wide=True),
        # The largest size of the serving range.
        _dvnd("search_1999", 1999),
        # The large configuration: 400 MB of distances, 64-bit latencies, a capped search.
        _dvnd("search_10000_wide", 10000, wide=True, iters=40),
        # A handful of starts of a few instances in one batch.
        _batch("batch_24", 6, 4, 100, 1000),
        # The batched configuration: 512 instances x 4 starts, n log-uniform in [100, 1000].
        _batch("batch_2048", 512, 4, 100, 1000),
        # A burst of requests at the serving loop, n log-uniform in [50, 2000], half uniform, half clustered.
        {"name": "serve_192", "kind": "serve", "requests": 192, "lo": 50, "hi": 2000},
        # A driver that walks the neighbourhoods one at a time (evaluate, then one pass of each; Or-opt-k last).
        {"name": "passes_1000", "kind": "passes", "n": 1000, "k": 4, "wide": False},
        # Multi-start: GRASP starts of one instance built on the device.
        {"name": "starts_512", "kind": "starts", "n": 1000, "count": 512, "alpha": 0.5},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["dvnd", "dvnd", "dvnd", "large", "batch", "serve", "passes", "starts"])
    if kind == "dvnd":
        c = _dvnd("", _log_int(rng, 20, 2300), wide=rng.random() < 0.3, mask=rng.choice([ALL, ALL, ALL, ALL, 0x12, 0x07]),
                  layout=rng.choice(["uniform", "clustered"]), rounded=rng.random() < 0.7)
    elif kind == "large":
        n = _log_int(rng, 2400, 9000)
        c = _dvnd("", n, wide=rng.random() < 0.7, iters=rng.randint(8, 40), layout=rng.choice(["uniform", "clustered"]))
    elif kind == "batch":
        lo = _log_int(rng, 40, 400)
        c = _batch("", _log_int(rng, 2, 200), rng.randint(1, 4), lo, min(1000, int(lo * (1.5 + 4 * rng.random()))),
                   layout=rng.choice(["uniform", "clustered"]))
    elif kind == "serve":
        lo = _log_int(rng, 50, 200)
        c = {"name": "", "kind": "serve", "requests": _log_int(rng, 4, 190), "lo": lo, "hi": _log_int(rng, 2 * lo, 2000)}
    elif kind == "passes":
        c = {"name": "", "kind": "passes", "n": _log_int(rng, 40, 2500), "k": rng.randint(1, 28), "wide": rng.random() < 0.3}
    else:
        c = {"name": "", "kind": "starts", "n": _log_int(rng, 50, 2000), "count": _log_int(rng, 4, 512),
             "alpha": round(0.05 + 0.9 * rng.random(), 2)}
    del c["name"]
    return c


def _sizes(count, lo, hi):
    """count sizes spread evenly over the logarithm of [lo, hi]."""
    return [int(v) for v in np.rint(np.exp(np.linspace(np.log(lo), np.log(hi), max(count, 2))[:count]))]


def _coords(layout, n, seed):
    return (workloads.uniform_instance if layout == "uniform" else workloads.clustered_instance)(n, seed)


def _request_layout(q):
    return "uniform" if q % 2 == 0 else "clustered"


def prepare(case, seed):
    kind, seed = case["kind"], int(seed)
    if kind == "dvnd":
        n = case["n"]
        p = mlpgpu.Problem.from_coords(*_coords(case["layout"], n, seed), dist_round=case["rounded"])
        return {"case": case, "solver": mlpgpu.Solver(p, wide=case["wide"]), "start": workloads.random_perm_tour(n, seed)}
    if kind == "batch":
        b = mlpgpu.Batch()
        for q, n in enumerate(_sizes(case["instances"], case["lo"], case["hi"])):
            p = mlpgpu.Problem.from_coords(*_coords(case["layout"], n, seed * 100_003 + q))
            for k in range(case["starts"]):
                b.add(p, workloads.random_perm_tour(n, seed * 100_003 + q * 8 + k))
        return {"case": case, "batch": b}
    if kind == "serve":
        reqs = []
        sizes = _sizes(case["requests"], case["lo"], case["hi"])
        for q, n in enumerate(np.random.default_rng(seed).permutation(sizes)):
            s = seed * 100_003 + q
            reqs.append((*_coords(_request_layout(q), int(n), s), workloads.random_perm_tour(int(n), s)))
        return {"case": case, "server": mlpgpu.Server(40 << 30, max_active=1024), "requests": reqs}
    n = case["n"]
    x, y = _coords("uniform", n, seed)
    p = mlpgpu.Problem.from_coords(x, y)
    if kind == "passes":
        s = mlpgpu.Solver(p, wide=case["wide"])
        return {"case": case, "solver": s, "start": workloads.random_perm_tour(n, seed)}
    return {"case": case, "problem": p, "seeds": np.random.default_rng(seed).integers(0, 1 << 32, case["count"], dtype=np.uint32)}


def _stats(dicts):
    return np.array([[d["cost"], d["iterations"], d["sweeps"], d["moves"], d["evals"], d["converged"]] for d in dicts],
                    np.int64)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "dvnd":
        s = state["solver"]
        s.set_tour(state["start"])
        st = s.dvnd(case["mask"], case["iters"])
        return {"stats": _stats([st]), "tour": s.tour()}
    if kind == "batch":
        b = state["batch"]
        b.reset()
        b.run()
        got = [b.result(j) for j in range(len(b.sizes))]
        return {"stats": _stats([st for _, st in got]), "tours": np.concatenate([t for t, _ in got])}
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(x, y, t) for x, y, t in state["requests"]]
        active = queued = 1
        while active or queued:
            active, queued = srv.step(8)
        srv.finished(len(ids))
        got = [srv.result(rid, len(t) - 1) for rid, (_, _, t) in zip(ids, state["requests"])]
        return {"stats": _stats([st for _, st, _ in got]), "tours": np.concatenate([t for t, _, _ in got])}
    if kind == "passes":
        s = state["solver"]
        s.set_tour(state["start"])
        first = [s.eval(nb) for nb in range(5)]
        moves, costs = [], []
        for nb in range(5):
            c, mv = s.pass_(nb)
            moves += mv
            costs.append(c)
        cand = s.eval_oropt(case["k"])
        c, mv = s.pass_oropt(case["k"])
        applied = np.full((4 * case["n"], 4), -1, np.int64)  # kept moves are independent: far fewer than 4 n
        applied[:len(moves) + len(mv)] = moves + mv
        return {"first_cost": [f[0] for f in first], "first_i": [f[1] for f in first], "first_j": [f[2] for f in first],
                "moves": applied, "costs": np.array(costs + [c], np.int64),
                "oropt": list(cand), "tour": s.tour()}
    return {"tours": state["problem"].random_tours(state["seeds"], case["alpha"])}


def _evals(n, mask=ALL):
    """Move evaluations of one sweep (the neighbourhood kernels' threads)."""
    size = n + 1
    per = [((size + 1) // 2 - 1) * (size - 4), ((size + 1) // 2) * (size - 3)] + [(size - k - 2) ** 2 for k in (1, 2, 3)]
    return sum(e for nb, e in enumerate(per) if (mask >> nb) & 1)


def work(case):
    """Distances (or coordinates) and starts read once, tours written once; about eight integer operations a move."""
    kind = case["kind"]
    if kind == "dvnd":
        n = case["n"]
        sweeps = min(case["iters"], n // 4 + 4)
        return {"bytes": 4 * n * n + 8 * n, "flops": 8 * sweeps * _evals(n, case["mask"])}
    if kind == "batch":
        ns = _sizes(case["instances"], case["lo"], case["hi"])
        return {"bytes": sum(4 * n * n + case["starts"] * 8 * n for n in ns),
                "flops": sum(8 * case["starts"] * (n // 4 + 4) * _evals(n) for n in ns)}
    if kind == "serve":
        ns = _sizes(case["requests"], case["lo"], case["hi"])
        return {"bytes": sum(16 * n + 4 * n * n for n in ns), "flops": sum(8 * (n // 4 + 4) * _evals(n) for n in ns)}
    n = case["n"]
    if kind == "passes":
        return {"bytes": 4 * n * n + 100 * n, "flops": 8 * (2 * _evals(n) + 2 * (n - case["k"]) ** 2)}
    # Each step of a start selects one of the remaining clients by rank.
    return {"bytes": 4 * n * n + 4 * n * case["count"], "flops": case["count"] * n * n // 2}


def exact(case, seed):
    """The per-block best deltas of the start tour from their definitions, in 64-bit whole numbers; searches, passes
    and the constructor return whole numbers that follow from long chains of decisions and have no such value."""
    if case["kind"] != "passes" or case["n"] > 1500:
        return None
    n = case["n"]
    x, y = (v.astype(np.int64) for v in _coords("uniform", n, int(seed)))
    d2 = ((x[:, None] - x[None, :]) ** 2 + (y[:, None] - y[None, :]) ** 2).astype(np.float32)
    dist = (np.sqrt(d2) + np.float32(0.5)).astype(np.int64)
    t = workloads.random_perm_tour(n, int(seed)).astype(np.int64)
    sz = n + 1
    e = np.zeros((sz + 8, sz + 8), np.int64)
    e[:sz, :sz] = dist[np.ix_(t, t)]
    w = np.zeros(sz + 8, np.int64)
    w[1:sz] = e[np.arange(sz - 1), np.arange(1, sz)]
    arrive, moment = np.cumsum(w), np.cumsum(np.arange(sz + 8) * w)
    first = []
    for nb in range(5):
        k = nb - 1
        blocks, threads = [((sz + 1) // 2 - 1, sz - 4), ((sz + 1) // 2, sz - 3)][nb] if nb < 2 else (sz - k - 2, sz - k - 2)
        by, ctx = np.arange(blocks)[:, None], np.arange(threads)[None, :]
        up = ctx >= by
        if nb == 0:
            i, j = np.where(up, by + 1, sz - by - 3), np.where(up, ctx + 3, sz - ctx - 2)
            d = ((sz - i) * (e[i - 1, j] - w[i]) + (sz - i - 1) * (e[j, i + 1] - w[i + 1])
                 + (sz - j) * (e[j - 1, i] - w[j]) + (sz - j - 1) * (e[i, j + 1] - w[j + 1]))
        elif nb == 1:
            i, j = np.where(up, ctx - by + 1, by - ctx), np.where(up, ctx + 2, sz - ctx - 2)
            d = ((sz - i) * (e[i - 1, j] - w[i]) + (sz - j - 1) * (e[i, j + 1] - w[j + 1])
                 + 2 * (moment[j] - moment[i]) - (i + j + 1) * (arrive[j] - arrive[i]))
        else:
            i, j = np.where(up, ctx - by + 1, sz - ctx - k - 1), np.where(up, ctx + 2, by - ctx)
            inner = (i - j) * (arrive[i + k - 1] - arrive[i])
            fwd = ((sz - i) * (e[i - 1, i + k] - w[i]) + (sz - j - k) * (e[i + k - 1, j + k] - w[j + k])
                   + (sz - j) * e[j + k - 1, i] - (sz - i - k) * w[i + k] + inner
                   + k * (arrive[j + k - 1] - arrive[i + k]))
            bwd = ((sz - j) * (e[j - 1, i] - w[j]) + (sz - i - k) * (e[i - 1, i + k] - w[i + k])
                   + (sz - j - k) * e[i + k - 1, j] - (sz - i) * w[i] + inner - k * (arrive[i - 1] - arrive[j]))
            d = np.where(up, fwd, bwd)
        first.append(d.min(axis=1))
    return {"first_cost": first, "first_i": None, "first_j": None, "moves": None, "costs": None, "oropt": None, "tour": None}
