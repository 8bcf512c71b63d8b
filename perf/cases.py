"""Performance cases: the solves and evaluations that programs have this
framework do, through its Python entry points (Model, Solver, Batch, Server).

Every case builds its instances from a seed.  `prepare` makes what a program
holds before the call (the models and the configured solver, batch or server),
`run` is one whole call with its results read back to the host.  Models follow
the framework's benchmark configurations (sparse Erdos-Renyi Ising models with
fields, random PUBO terms of orders 1-4, +-J lattices, weighted random 3-SAT),
with sweep counts cut so that a pass stays below two seconds.
"""
import math

import numpy as np

from qiotoolkit_gb300 import Batch, Model, Server, Solver
from qiotoolkit_gb300 import instances as I

SA = "simulatedannealing.qiotoolkit"
PT = "paralleltempering.qiotoolkit"
PA = "populationannealing.cpu"


def listed():
    return [
        # the smallest call: a tiny Ising model, few restarts, a short anneal
        # (latency, launches and copies)
        {"name": "sa_small", "kind": "sa_ising", "n": 64, "edges": 192, "restarts": 8, "sweeps": 100,
         "integer": False, "rng": "replay"},
        # simulated annealing on a sparse random Ising model with fields
        {"name": "sa_ising", "kind": "sa_ising", "n": 1000, "edges": 3000, "restarts": 64, "sweeps": 1000,
         "integer": False, "rng": "replay"},
        # parallel tempering on a random PUBO, a swap after every sweep
        {"name": "pt_pubo", "kind": "pt_pubo", "n": 4096, "terms": 20000, "temps": 32, "restarts": 16,
         "sweeps": 100, "integer": False, "rng": "replay"},
        # parallel tempering on weighted random 3-SAT, every variable per sweep
        {"name": "pt_maxsat", "kind": "pt_maxsat", "n": 1000, "temps": 8, "restarts": 8, "sweeps": 200,
         "integer": False, "rng": "replay"},
        # population annealing on a periodic +-J square lattice, counter
        # streams, a constant population (so that its size is the case's); the
        # whole population is read back
        {"name": "pa_square", "kind": "pa_square", "L": 128, "population": 2048, "steps": 10, "spr": 10},
        # many independent instances in one batch: cubic +-J lattices
        {"name": "batch_cubic", "kind": "batch_cubic", "count": 96, "lmin": 4, "lmax": 20, "restarts": 16,
         "sweeps": 100, "rng": "replay"},
        # the same for many-body models: random PUBO instances of mixed size
        {"name": "batch_pubo", "kind": "batch_pubo", "count": 96, "nmin": 100, "nmax": 2000, "restarts": 16,
         "sweeps": 100, "rng": "replay"},
        # serving: a burst of mixed requests (three kinds of model, annealing
        # and tempering) through one server
        {"name": "serving", "kind": "serving", "count": 24, "nmax": 2000, "smin": 200, "smax": 600},
        # tabu search, many restarts
        {"name": "tabu_ising", "kind": "tabu", "n": 1000, "edges": 3000, "restarts": 1216, "sweeps": 200,
         "tenure": 20, "integer": False},
        # quantum Monte Carlo with the reference's replayed streams
        {"name": "qmc_ising", "kind": "qmc", "n": 1000, "edges": 3000, "restarts": 16, "slices": 32,
         "sweeps": 50, "integer": False, "rng": "replay"},
        # substochastic Monte Carlo, a population resampled every step
        {"name": "ssmc_ising", "kind": "ssmc", "n": 1000, "edges": 3000, "population": 4096, "sweeps": 50,
         "spw": 4, "integer": False, "rng": "counter"},
        # the per-state contract: costs and cost differences of given states
        {"name": "states_pubo", "kind": "states", "n": 4096, "terms": 20000, "states": 1024, "integer": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sa_ising", "sa_ising", "pt_pubo", "pt_maxsat", "pa_square", "batch_cubic", "batch_pubo",
                       "serving", "tabu", "qmc", "ssmc", "states"])
    mode = rng.choice(["replay", "replay", "counter"])
    integer = rng.random() < 0.3
    n = _log(rng, 64, 2000)
    edges = int(n * rng.uniform(1.5, 4.0))
    if kind == "sa_ising":
        restarts = _log(rng, 4, 512)
        sweeps = min(1000, max(20, int(6e7 / (n * max(restarts, 64)))))
        return {"kind": kind, "n": n, "edges": edges, "restarts": restarts, "sweeps": sweeps, "integer": integer,
                "rng": mode}
    if kind == "pt_pubo":
        n = _log(rng, 100, 4096)
        return {"kind": kind, "n": n, "terms": int(n * rng.uniform(2.0, 5.0)), "temps": rng.randint(4, 32),
                "restarts": rng.randint(1, 16), "sweeps": rng.randint(20, 100), "integer": integer, "rng": mode}
    if kind == "pt_maxsat":
        return {"kind": kind, "n": _log(rng, 100, 3000), "temps": rng.randint(4, 16), "restarts": rng.randint(1, 8),
                "sweeps": rng.randint(20, 60), "integer": integer, "rng": mode}
    if kind == "pa_square":
        return {"kind": kind, "L": rng.randint(64, 160), "population": _log(rng, 256, 1250),
                "steps": rng.randint(4, 10), "spr": rng.randint(2, 10)}
    if kind == "batch_cubic":
        lmin = rng.randint(3, 8)
        return {"kind": kind, "count": rng.randint(8, 96), "lmin": lmin, "lmax": rng.randint(lmin + 2, 18),
                "restarts": rng.randint(4, 16), "sweeps": rng.randint(20, 100), "rng": mode}
    if kind == "batch_pubo":
        return {"kind": kind, "count": rng.randint(8, 96), "nmin": 100, "nmax": _log(rng, 300, 2000),
                "restarts": rng.randint(4, 16), "sweeps": rng.randint(20, 100), "rng": mode}
    if kind == "serving":
        return {"kind": kind, "count": rng.randint(4, 24), "nmax": _log(rng, 200, 2000), "smin": rng.randint(50, 200),
                "smax": rng.randint(201, 500)}
    if kind == "tabu":
        return {"kind": kind, "n": n, "edges": edges, "restarts": _log(rng, 16, 1216), "sweeps": rng.randint(50, 300),
                "tenure": rng.randint(5, 40), "integer": integer}
    if kind == "qmc":
        return {"kind": kind, "n": _log(rng, 64, 1000), "edges": 0, "restarts": rng.randint(2, 16),
                "slices": rng.randint(4, 48), "sweeps": rng.randint(10, 40), "integer": integer, "rng": mode}
    if kind == "ssmc":
        return {"kind": kind, "n": n, "edges": edges, "population": _log(rng, 128, 4096),
                "sweeps": rng.randint(20, 50), "spw": rng.randint(1, 6), "integer": integer, "rng": mode}
    n = _log(rng, 64, 4096)
    return {"kind": kind, "n": n, "terms": int(n * rng.uniform(2.0, 5.0)), "states": _log(rng, 16, 1024),
            "integer": integer}


# ---- instances ------------------------------------------------------------
def _rows(rng, n, order, count):
    """count rows of `order` distinct variables below n."""
    out = rng.integers(0, n, (count, order))
    while True:
        s = np.sort(out, 1)
        bad = np.flatnonzero((s[:, 1:] == s[:, :-1]).any(1))
        if not len(bad):
            return s
        out = s
        out[bad] = rng.integers(0, n, (len(bad), order))


def _cover(rng, ids, n):
    """Every variable below n in some term: each missing one takes the place of
    a variable that occurs again elsewhere (so that a size is a size)."""
    count = np.bincount(ids, minlength=n)
    for v in np.flatnonzero(count == 0):
        while True:
            p = int(rng.integers(0, len(ids)))
            if count[ids[p]] > 1:
                break
        count[ids[p]] -= 1
        count[v] = 1
        ids[p] = v
    return ids


def _pubo(n, terms, seed, integer, orders=(1, 2, 3, 4), probs=(0.1, 0.5, 0.3, 0.1)):
    """Random PUBO terms: orders by `probs`, distinct variables, N(0,1)
    weights (integer: nonzero weights in -3 .. 3)."""
    rng = np.random.default_rng(seed)
    o = rng.choice(orders, size=terms, p=probs)
    off = np.zeros(terms + 1, np.int64)
    off[1:] = np.cumsum(o)
    ids = np.zeros(off[-1], np.int32)
    for k in orders:
        at = np.flatnonzero(o == k)
        if len(at):
            ids[off[at][:, None] + np.arange(k)] = _rows(rng, n, k, len(at))
    ids = _cover(rng, ids, n)
    coef = rng.choice([-3.0, -2.0, -1.0, 1.0, 2.0, 3.0], terms) if integer else rng.standard_normal(terms)
    return off, ids, coef


def _ising(n, edges, seed, integer):
    """Erdos-Renyi +-1 couplings with one field per spin (integer: +-1 fields)."""
    edges = min(edges or 3 * n, n * (n - 1) // 3)
    off, ids, coef = I.er_ising(n, edges, seed=seed)
    if integer:
        coef = np.where(coef < 0, -1.0, 1.0)
    return off, ids, coef


def _maxsat(n, seed, integer, ratio=4.2):
    """Weighted random 3-SAT, weights uniform in [1, 10]."""
    rng = np.random.default_rng(seed)
    m = int(round(ratio * n))
    ids = (_cover(rng, _rows(rng, n, 3, m).ravel(), n) + 1) * rng.choice([-1, 1], 3 * m)
    coef = rng.integers(1, 11, m).astype(float) if integer else rng.uniform(1.0, 10.0, m)
    return 3 * np.arange(m + 1, dtype=np.int64), ids.astype(np.int32), coef


def _requests(c, seed):
    rng = np.random.default_rng(c["count"])  # the mix is the case's, the models the seed's
    out = []
    for i in range(c["count"]):
        kind = i % 3
        n = int(np.exp(rng.uniform(np.log(100), np.log(c["nmax"]))))
        s = seed + i
        if kind == 0:
            off, ids, coef = I.er_ising_gauss(n, float(rng.uniform(4, 16)), seed=s)
            k, inst = "ising", (off, _cover(np.random.default_rng(s), ids, n), coef)
        elif kind == 1:
            k, inst = "pubo", _pubo(n, 3 * n, s, False, (1, 2, 3), (1 / 3, 1 / 3, 1 / 3))
        else:
            k, inst = "maxsat", _maxsat(n, s, False)
        p = {"seed": i, "sweeps": int(rng.integers(c["smin"], c["smax"] + 1))}
        if rng.integers(0, 2):
            p["temperatures"] = {"type": "geometric", "initial": 0.1, "final": 3.0, "count": 8}
            out.append((k, inst, PT, p))
        else:
            p.update(restarts=8, beta_start=0.1, beta_stop=3.0)
            out.append((k, inst, SA, p))
    return out


def _model(kind, inst):
    off, ids, coef = inst
    return Model(kind, off=off, ids=ids, coef=coef)


def _sa_params(c, seed):
    return {"seed": seed, "sweeps": c["sweeps"], "restarts": c["restarts"], "beta_start": 0.1, "beta_stop": 5.0,
            "rng_mode": c["rng"]}


def prepare(case, seed):
    c, kind = case, case["kind"]
    st = {"kind": kind}
    pseed = seed % 1000003
    if kind == "sa_ising":
        m = _model("ising", _ising(c["n"], c["edges"], seed, c["integer"]))
        st["solver"] = Solver(m, SA, _sa_params(c, pseed))
    elif kind in ("pt_pubo", "pt_maxsat"):
        p = {"seed": pseed, "sweeps": c["sweeps"], "restarts": c["restarts"], "rng_mode": c["rng"],
             "temperatures": {"type": "geometric", "initial": 0.05, "final": 3.0, "count": c["temps"]}}
        if kind == "pt_pubo":
            m = _model("pubo", _pubo(c["n"], c["terms"], seed, c["integer"]))
        else:
            m = _model("maxsat", _maxsat(c["n"], seed, c["integer"]))
            p["maxsat_full_sweep"] = True
        st["solver"] = Solver(m, PT, p)
    elif kind == "pa_square":
        m = _model("ising", I.square_pm_j(c["L"], seed=seed))
        st["solver"] = Solver(m, PA, {"seed": pseed, "sweeps": c["steps"], "population": c["population"],
                                      "beta_start": 0.0, "beta_stop": 3.0, "sweeps_per_replica": c["spr"],
                                      "constant_population": True, "rng_mode": "counter", "threads": 16})
    elif kind in ("batch_cubic", "batch_pubo"):
        rng = np.random.default_rng(c["count"])  # the sizes are the case's, the models the seed's
        st["models"] = []
        for i in range(c["count"]):
            if kind == "batch_cubic":
                # the range's largest instance is always among them
                L = c["lmax"] if i == 0 else int(rng.integers(c["lmin"], c["lmax"] + 1))
                inst, k = I.cubic_pm_j(L, seed=seed + i), "ising"
            else:
                n = c["nmax"] if i == 0 else int(np.exp(rng.uniform(np.log(c["nmin"]), np.log(c["nmax"]))))
                inst, k = _pubo(n, 3 * n, seed + i, False), "pubo"
            st["models"].append(_model(k, inst))
        st["batch"] = Batch(st["models"], SA, {"seed": pseed, "sweeps": c["sweeps"], "restarts": c["restarts"],
                                               "beta_start": 0.1, "beta_stop": 3.0, "rng_mode": c["rng"]})
    elif kind == "serving":
        st["requests"] = [(_model(k, inst), t, p) for k, inst, t, p in _requests(c, seed)]
        # a serving program has its models on the device before the burst
        for m, _, _ in st["requests"]:
            m.calculate_cost(np.zeros(m.n_vars, np.uint8))
        st["server"] = Server(memory_budget_bytes=4 << 30)
    elif kind == "tabu":
        m = _model("ising", _ising(c["n"], c["edges"], seed, c["integer"]))
        st["solver"] = Solver(m, "tabu.qiotoolkit", {"seed": pseed, "sweeps": c["sweeps"], "restarts": c["restarts"],
                                                     "tabu_tenure": c["tenure"]})
    elif kind == "qmc":
        m = _model("ising", _ising(c["n"], c["edges"], seed, c["integer"]))
        st["solver"] = Solver(m, "quantummontecarlo.qiotoolkit",
                              {"seed": pseed, "sweeps": c["sweeps"], "restarts": c["restarts"],
                               "trotter_number": c["slices"], "beta_start": 1.0, "beta_stop": 5.0,
                               "transverse_field_low": 0.0, "transverse_field_high": 3.0, "rng_mode": c["rng"]})
    elif kind == "ssmc":
        m = _model("ising", _ising(c["n"], c["edges"], seed, c["integer"]))
        st["solver"] = Solver(m, "substochasticmontecarlo.cpu",
                              {"seed": pseed, "sweeps": c["sweeps"], "target_population": c["population"],
                               "steps_per_walker": c["spw"], "threads": 16, "rng_mode": c["rng"]})
    else:
        st["model"] = _model("pubo", _pubo(c["n"], c["terms"], seed, c["integer"]))
        st["states"], st["vars"] = _given(st["model"].n_vars, c, seed)
    return st


def _given(n_vars, c, seed):
    rng = np.random.default_rng(seed + 1)
    return rng.integers(0, 2, (c["states"], n_vars), dtype=np.uint8), rng.integers(0, n_vars, c["states"])


def _answer(result):
    """A result document's cost and configuration as numbers."""
    s = result["solutions"]
    conf = s["configuration"]
    return {"cost": float(s["cost"]), "vars": np.fromiter((int(k) for k in conf), np.int64, len(conf)),
            "values": np.fromiter(conf.values(), np.int64, len(conf))}


def _joined(answers):
    return {"cost": np.array([a["cost"] for a in answers]), "vars": np.concatenate([a["vars"] for a in answers]),
            "values": np.concatenate([a["values"] for a in answers])}


def run(state):
    kind = state["kind"]
    if kind in ("batch_cubic", "batch_pubo"):
        b = state["batch"]
        b.run()
        out = _joined([_answer(b.result(i)) for i in range(len(state["models"]))])
        out["lowest"] = b.lowest()
        return out
    if kind == "serving":
        srv = state["server"]
        rids = [srv.submit(m, t, p) for m, t, p in state["requests"]]
        got = [_answer(srv.wait(r)) for r in rids]
        for r in rids:
            srv.forget(r)
        return _joined(got)
    if kind == "states":
        m = state["model"]
        return {"cost": m.calculate_cost(state["states"]),
                "diff": m.calculate_cost_difference(state["states"], state["vars"])}
    s = state["solver"]
    s.init().run()
    out = s.replicas()
    if kind in ("pt_pubo", "pt_maxsat"):
        out["observables"] = np.nan_to_num(s.pt_observables(), nan=-1.0)
    return {k: (v.astype(np.int64) if v.dtype == np.uint64 else v) for k, v in out.items()}


# ---- what a pass cannot do without -------------------------------------------
# flops: ten per flip attempt (field, threshold, draw and comparison); bytes:
# the model read once and the walkers' results written once.
def work(case):
    c, kind = case, case["kind"]

    def of(n, inc, terms, walkers, attempts):
        return {"bytes": 8 * inc + 12 * terms + walkers * (2 * n / 8 + 32), "flops": 10 * attempts}

    if kind in ("sa_ising", "tabu", "qmc", "ssmc"):
        n, e = c["n"], c["edges"] or 3 * c["n"]
        walkers = {"qmc": c["restarts"] * c.get("slices", 1) if kind == "qmc" else 0,
                   "ssmc": c.get("population", 0)}.get(kind, c.get("restarts", 0))
        per = {"ssmc": c.get("spw", 0)}.get(kind, n)
        return of(n, n + 2 * e, n + e, walkers, walkers * c["sweeps"] * per)
    if kind == "pt_pubo":
        w = c["temps"] * c["restarts"]
        return of(c["n"], 2.4 * c["terms"], c["terms"], w, w * c["sweeps"] * c["n"])
    if kind == "pt_maxsat":
        w = c["temps"] * c["restarts"]
        return of(c["n"], 12.6 * c["n"], 4.2 * c["n"], w, w * c["sweeps"] * c["n"])
    if kind == "pa_square":
        n = c["L"] ** 2
        return of(n, 4 * n, 2 * n, c["population"], c["population"] * c["steps"] * c["spr"] * n)
    if kind == "batch_cubic":
        n = sum(L**3 for L in range(c["lmin"], c["lmax"] + 1)) / (c["lmax"] + 1 - c["lmin"]) * c["count"]
        return of(n, 6 * n, 3 * n, c["restarts"], c["restarts"] * c["sweeps"] * n)
    if kind == "batch_pubo":
        n = (c["nmax"] - c["nmin"]) / math.log(c["nmax"] / c["nmin"]) * c["count"]
        return of(n, 7.2 * n, 3 * n, c["restarts"], c["restarts"] * c["sweeps"] * n)
    if kind == "serving":
        n = (c["nmax"] - 100) / math.log(c["nmax"] / 100) * c["count"]
        # a 3-SAT sweep is one attempt: two requests in three sweep all variables
        return of(n, 9 * n, 4 * n, 8, 8 * (c["smin"] + c["smax"]) / 2 * n * 2 / 3)
    return {"bytes": 2 * c["states"] * c["n"] + 32 * c["terms"] + 24 * c["states"],
            "flops": c["states"] * (2.4 + 1) * c["terms"]}


# ---- exact values -----------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "states":
        return _exact_states(case, seed)
    if case["kind"] == "sa_ising" and case["rng"] == "replay" and case["restarts"] * case["sweeps"] * case["n"] < 1e6:
        return _exact_sa(case, seed)
    return None


def _first_appearance(ids):
    """Internal ids: names numbered by first appearance."""
    names, first = np.unique(ids, return_index=True)
    rank = np.argsort(np.argsort(first))
    return rank[np.searchsorted(names, ids)], len(names)


def _exact_states(c, seed):
    off, ids, coef = _pubo(c["n"], c["terms"], seed, c["integer"])
    v, n = _first_appearance(ids)
    states, at = _given(n, c, seed)
    x = np.ascontiguousarray((1 - states).T)  # a true state bit is the value 0

    def cost(x):
        total = np.zeros(x.shape[1])
        for t in range(len(coef)):
            live = x[v[off[t]]]
            for k in range(off[t] + 1, off[t + 1]):
                live = live & x[v[k]]
            total += coef[t] * live
        return total

    # a flip's difference: the terms of the variable whose other members are 1
    q = np.arange(len(at))
    terms_of = [[] for _ in range(n)]
    for t in range(len(coef)):
        for k in range(off[t], off[t + 1]):
            terms_of[v[k]].append(t)
    diff = np.zeros(len(at))
    for i in q:
        d = 0.0
        for t in terms_of[at[i]]:
            if all(x[w, i] for w in v[off[t]:off[t + 1]] if w != at[i]):
                d += coef[t]
        diff[i] = d if not x[at[i], i] else -d
    return {"cost": cost(x), "diff": diff}


def _exact_sa(c, seed):
    """The reference's annealing chain replayed: PCG streams, the ordered
    sweep, the ln-table Metropolis decision (utils/random_generator.cc,
    markov/walker.h, markov/metropolis.h)."""
    off, ids, coef = _ising(c["n"], c["edges"], seed, c["integer"])
    v, n = _first_appearance(ids)
    v = v.tolist()
    terms = [[v[k] for k in range(off[t], off[t + 1])] for t in range(len(coef))]
    cf = coef.tolist()
    rows = [[] for _ in range(n)]
    for t, mem in enumerate(terms):
        for u in mem:
            rows[u].append(([w for w in mem if w != u], cf[t]))
    mult, inc, full = 6364136223846793005, 1442695040888963407, (1 << 64) - 1
    ln = [[-math.inf if b == 0 else math.log(b / 256.0 ** (r + 1)) for b in range(256)] for r in range(4)]

    def seeded(s):
        return ((s + inc) * mult + inc) & full

    def out(s):
        x = (((s >> 18) ^ s) >> 27) & 0xFFFFFFFF
        r = s >> 59
        return ((x >> r) | (x << ((32 - r) & 31))) & 0xFFFFFFFF

    master = seeded(seed % 1000003)
    res = {k: [] for k in ("cost", "lowest", "attempts", "accepts", "lowest_states", "states")}
    sweeps = c["sweeps"]
    stop = max(1, sweeps - 1)
    for _ in range(c["restarts"]):
        s = seeded(out(master))
        master = (master * mult + inc) & full
        spin = []
        for _w in range((n + 31) // 32):
            word = out(s)
            s = (s * mult + inc) & full
            spin += [(word >> b) & 1 for b in range(32)]
        spin = spin[:n]
        cost = 0.0
        for t, mem in enumerate(terms):
            cost += -cf[t] if sum(spin[u] for u in mem) & 1 else cf[t]
        low, low_spin, acc = cost, list(spin), 0
        for k in range(sweeps):
            beta = 0.1 + min(1.0, k / stop) * (5.0 - 0.1)
            for i in range(n):
                d = 0.0
                for others, w in rows[i]:
                    p = spin[i]
                    for u in others:
                        p ^= spin[u]
                    d += -w if p else w
                d = 2.0 * -d
                ok = d <= 0
                if not ok:
                    b, r = 0, -1
                    while b == 0 and r < 3:
                        g = out(s)
                        s = (s * mult + inc) & full
                        b, r = g & 255, r + 1
                    if b == 0:
                        ok = True
                    elif b > 1:
                        y0 = ln[r][b - 1]
                        ok = y0 + (g >> 8) / 16777214.0 * (ln[r][b] - y0) < d * -beta
                if ok:
                    spin[i] ^= 1
                    acc += 1
                    cost += d
                    if cost < low:
                        low, low_spin = cost, list(spin)
        for key, val in (("cost", cost), ("lowest", low), ("attempts", sweeps * n), ("accepts", acc),
                         ("lowest_states", low_spin), ("states", spin)):
            res[key].append(val)
    kinds = {"cost": np.float64, "lowest": np.float64, "attempts": np.int64, "accepts": np.int64,
             "lowest_states": np.uint8, "states": np.uint8}
    return {k: np.array(x, kinds[k]) for k, x in res.items()}
