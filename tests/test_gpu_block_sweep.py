"""Edges of the block-decided sweep (csrc/fields.cu) against the oracle, bit for
bit (GPU required): variables around a block of 32, a walker's last and only
block, terms inside one block and across its border, more in-block terms per
lane than a chunk holds, terms of more members than a byte's bits or a record's
fields, rows wider than a staged block, draws that no attempt takes (an
infinite beta), more walkers than fit the chip at once, and sweeps cut into
launches of one."""
import numpy as np
import pytest

import qiotoolkit_gb300 as q
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SA = "simulatedannealing.qiotoolkit"


def terms(n, sizes, count, seed, span=None, integer=False, hub=0):
    """`count` terms of the given sizes over n variables, each within a run of
    `span` ids; `hub` further terms on variable n // 2; every variable in one."""
    rng = np.random.default_rng(seed)
    out = [[v] for v in range(n)]
    for _ in range(count):
        k = min(int(rng.choice(sizes)), n)
        lo = 0 if span is None else int(rng.integers(0, max(1, n - span + 1)))
        hi = n if span is None else min(n, lo + max(span, k))
        out.append(sorted((lo + rng.choice(hi - lo, min(k, hi - lo), replace=False)).tolist()))
    for _ in range(hub):
        out.append(sorted({n // 2, *rng.choice(n, 2, replace=False).tolist()}))
    out = sorted({tuple(t) for t in out})
    coef = rng.choice([-2.0, -1.0, 1.0, 3.0], len(out)) if integer else rng.normal(size=len(out))
    return O.flatten_terms([(float(c), list(t)) for c, t in zip(coef, out)])


def clauses(n, seed, **kw):
    """The same with random signs, ids from 1 and positive weights."""
    off, ids, coef = terms(n, seed=seed, **kw)
    sign = np.random.default_rng(seed + 1).choice([-1, 1], len(ids))
    return off, (np.asarray(ids) + 1) * sign, np.abs(coef)


CASES = {  # kind, instance, restarts, beta_stop
    **{f"pair_{n}": ("ising", lambda n=n: terms(n, [2], 3 * n, n), 5, 3.0) for n in (2, 31, 32, 33, 64, 65)},
    **{f"pubo_{n}": ("pubo", lambda n=n: terms(n, [2, 3, 4], 4 * n, n), 5, 3.0) for n in (4, 32, 33, 97)},
    "pair_dense_block": ("ising", lambda: terms(70, [2], 700, 1, span=36, integer=True), 6, 2.0),
    "pair_wide_rows": ("ising", lambda: terms(200, [2], 300, 2, hub=150), 6, 2.0),
    "parity_block": ("ising", lambda: terms(90, [3, 4], 400, 3, span=40), 6, 3.0),
    "parity_large": ("ising", lambda: terms(120, [2, 5, 9, 12], 300, 4), 6, 3.0),
    "parity_large_int": ("ising", lambda: terms(120, [2, 6, 10], 300, 5, span=48, integer=True), 6, 3.0),
    "pubo_block": ("pubo", lambda: terms(80, [2, 3, 5], 500, 6, span=34), 6, 3.0),
    "pubo_block_int": ("pubo", lambda: terms(80, [2, 3, 6], 500, 7, span=34, integer=True), 6, 3.0),
    "pubo_large": ("pubo", lambda: terms(130, [1, 4, 7, 9, 14], 400, 8), 6, 3.0),
    "pubo_wide_rows": ("pubo", lambda: terms(260, [2, 3], 500, 9, hub=180), 6, 3.0),
    "pubo_widest_rows": ("pubo", lambda: terms(600, [2], 300, 15, hub=253), 4, 3.0),
    "sat_wide_block": ("maxsat", lambda: clauses(64, 16, sizes=[5, 6, 20], count=150, span=40), 6, 3.0),
    "sat_signs": ("maxsat", lambda: clauses(75, 10, sizes=[2, 3, 5], count=400, span=38), 6, 3.0),
    "sat_large": ("maxsat", lambda: clauses(100, 11, sizes=[3, 9, 11], count=300, integer=True), 6, 3.0),
    "cold": ("ising", lambda: terms(100, [2], 300, 12), 4, np.inf),
    "cold_pubo": ("pubo", lambda: terms(100, [2, 3], 300, 13), 4, np.inf),
    "waves": ("pubo", lambda: terms(60, [2, 3], 150, 14), 1300, 2.0),
}


@pytest.mark.parametrize("mode", ["replay", "counter"])
@pytest.mark.parametrize("name", list(CASES))
def test_block_sweep_edges(name, mode):
    kind, make, restarts, stop = CASES[name]
    inst = make()
    g = q.Model(kind, off=inst[0], ids=inst[1], coef=inst[2])
    o = O.Model(kind, off=inst[0], ids=inst[1], coef=inst[2])
    temps = np.isinf(stop)  # a temperature of zero
    params = {"seed": 3, "sweeps": 25, "restarts": restarts, "rng_mode": mode, "kernel": "fields",
              "maxsat_full_sweep": True, "cost_limit": -1e300}
    if restarts > 100:
        del params["cost_limit"]  # one launch for all sweeps
    sched = ("linear", 2.0, 0.0) if temps else ("linear", 0.1, stop)
    params.update({"schedule": {"type": "linear", "initial": 2.0, "final": 0.0}} if temps else
                  {"beta_start": 0.1, "beta_stop": stop})
    s = q.Solver(g, SA, {"params": params}).init().run()
    assert s.stats().sweep_kernel == 8
    r = O.run(o, "sa", seed=3, step_limit=25, restarts=restarts, sched=sched, use_inverse=not temps,
              rng_mode=mode, threads=8, full_maxsat_sweep=True)
    out = s.replicas()
    for key in ("cost", "lowest", "attempts", "accepts", "states", "lowest_states"):
        np.testing.assert_array_equal(out[key], getattr(r, key), err_msg=key)


@pytest.mark.parametrize("mode", ["replay", "counter"])
@pytest.mark.parametrize("kernel", ["auto", "fields"])
def test_batches_of_every_form(kernel, mode):
    """One queue per kind of model (pair, many-body and counter models, integer
    and FP64), small and large models behind one another on a walker's slot:
    every instance equals its plain windowed solve."""
    models = [q.Model("ising", off=t[0], ids=t[1], coef=t[2]) for t in (
        terms(400, [2], 900, 21), terms(33, [2], 60, 22), terms(380, [2], 800, 23, integer=True),
        terms(90, [2, 3, 4], 200, 24), terms(64, [2, 9], 150, 25, integer=True))]
    models += [q.Model("pubo", off=t[0], ids=t[1], coef=t[2]) for t in (
        terms(200, [2, 3, 4], 600, 26), terms(40, [2, 3], 100, 27, hub=40), terms(70, [2, 10], 90, 28, integer=True))]
    params = {"seed": 6, "sweeps": 12, "restarts": 9, "beta_start": 0.1, "beta_stop": 2.0, "rng_mode": mode}
    b = q.Batch(models, SA, {"params": dict(params, kernel=kernel)}).run()
    first = [b.result(i)["solutions"] for i in range(len(models))]
    for i, m in enumerate(models):
        plain = q.Solver(m, SA, {"params": dict(params, kernel="warp")}).init().run().result()
        assert first[i] == plain["solutions"], i
    assert [b.run().result(i)["solutions"] for i in range(len(models))] == first
    pairs = q.Batch(models[:2], SA, {"params": dict(params, kernel=kernel)}).run()
    assert pairs.stats().kernel == 1 and [pairs.result(i)["solutions"] for i in range(2)] == first[:2]


@pytest.mark.parametrize("mode", ["replay", "counter"])
@pytest.mark.parametrize("integer", [True, False])
@pytest.mark.parametrize("n", [5, 6, 32, 37, 64, 96, 200, 254])
def test_dense_pair_blocks(n, integer, mode):
    """Complete graphs, some couplings twice: a variable has four earlier members in
    its block (n = 5), five, or all; staged blocks and ones too large for that."""
    rng = np.random.default_rng(n)
    rows = [[v] for v in range(n) if v % 3] + [[a, b] for a in range(n) for b in range(a + 1, n)]
    rows += [rows[i] for i in rng.integers(0, len(rows), 3) if n < 250]
    coef = rng.choice([-1.0, 1.0], len(rows)) if integer else rng.normal(size=len(rows))
    off, ids, coef = O.flatten_terms([(float(c), r) for c, r in zip(coef, rows)])
    params = {"seed": 4, "sweeps": 30, "restarts": 5, "beta_start": 0.02, "beta_stop": 1.0, "rng_mode": mode,
              "kernel": "fields"}
    s = q.Solver(q.Model("ising", off=off, ids=ids, coef=coef), SA, {"params": params}).init().run()
    assert s.stats().sweep_kernel == 8
    r = O.run(O.Model("ising", off=off, ids=ids, coef=coef), "sa", seed=4, step_limit=30, restarts=5,
              sched=("linear", 0.02, 1.0), rng_mode=mode, threads=8)
    out = s.replicas()
    for key in ("cost", "lowest", "attempts", "accepts", "states", "lowest_states"):
        np.testing.assert_array_equal(out[key], getattr(r, key), err_msg=key)


SHARED = {  # models whose chunks are so large that a block's walkers share their buffers
    "pair": ("ising", lambda: terms(200, [2], 16000, 31)),
    "pair_int": ("ising", lambda: terms(130, [2], 7000, 32, integer=True)),
    "hub": ("ising", lambda: terms(320, [2], 600, 33, hub=240)),
    "pubo": ("pubo", lambda: terms(300, [2, 3], 500, 34, hub=240)),
    "pubo_int": ("pubo", lambda: terms(96, [2], 3500, 35, integer=True)),
}


@pytest.mark.parametrize("mode", ["replay", "counter"])
@pytest.mark.parametrize("restarts", [153, 305, 609, 1217])
@pytest.mark.parametrize("name", list(SHARED))
def test_shared_chunk_buffers(name, restarts, mode):
    """Blocks of two to eight walkers on the same buffers, the last ones not full."""
    kind, make = SHARED[name]
    inst = dict(zip(("off", "ids", "coef"), make()))
    params = {"seed": 9, "sweeps": 6, "restarts": restarts, "beta_start": 0.05, "beta_stop": 1.0, "rng_mode": mode,
              "kernel": "fields"}
    s = q.Solver(q.Model(kind, **inst), SA, {"params": params}).init().run()
    r = O.run(O.Model(kind, **inst), "sa", seed=9, step_limit=6, restarts=restarts, sched=("linear", 0.05, 1.0),
              rng_mode=mode, threads=8)
    out = s.replicas()
    for key in ("cost", "lowest", "attempts", "accepts", "states", "lowest_states"):
        np.testing.assert_array_equal(out[key], getattr(r, key), err_msg=key)


def _rows_of(n, degree, sizes, seed, integer=False):
    """Variables 0, 3, 6, ... with `degree` terms each, the others fewer."""
    rng = np.random.default_rng(seed)
    out = {(v,) for v in range(n)}
    count = np.ones(n, int)
    for v in range(0, n, 3):
        while count[v] < degree:
            others = rng.choice(np.setdiff1d(np.arange(n), np.arange(0, n, 3)), int(rng.choice(sizes)) - 1, replace=False)
            t = tuple(sorted({v, *others.tolist()}))
            if t not in out and count[list(others)].max() < 250:
                out.add(t)
                count[list(t)] += 1
    out = sorted(out)
    coef = rng.choice([-2.0, -1.0, 1.0, 3.0], len(out)) if integer else rng.normal(size=len(out))
    return O.flatten_terms([(float(c), list(t)) for c, t in zip(coef, out)])


@pytest.mark.parametrize("mode", ["replay", "counter"])
@pytest.mark.parametrize("kind,n,degree,sizes", [
    ("pubo", 40, 31, [3]), ("pubo", 40, 32, [3]), ("pubo", 40, 33, [3]), ("pubo", 33, 34, [3, 6]), ("pubo", 60, 90, [3, 4]),
    ("pubo", 290, 190, [2]), ("ising", 40, 32, [3]), ("ising", 40, 33, [3]), ("ising", 70, 64, [3, 4, 7])])
def test_rows_wider_than_the_masks(kind, n, degree, sizes, mode):
    """FP64 rows around 32 terms, the widest that a flip's log entry has masks for."""
    inst = dict(zip(("off", "ids", "coef"), _rows_of(n, degree, sizes, n + degree)))
    for stop in (1.0, 6.0):
        params = {"seed": 2, "sweeps": 40, "restarts": 7, "beta_start": 0.01, "beta_stop": stop, "rng_mode": mode,
                  "kernel": "fields"}
        s = q.Solver(q.Model(kind, **inst), SA, {"params": params}).init().run()
        assert s.stats().sweep_kernel == 8
        r = O.run(O.Model(kind, **inst), "sa", seed=2, step_limit=40, restarts=7, sched=("linear", 0.01, stop),
                  rng_mode=mode, threads=8)
        out = s.replicas()
        for key in ("cost", "lowest", "attempts", "accepts", "states", "lowest_states"):
            np.testing.assert_array_equal(out[key], getattr(r, key), err_msg=key)


@pytest.mark.parametrize("mode", ["replay", "counter"])
def test_batch_with_wide_and_narrow_rows(mode):
    """One queue for models with rows that have masks and rows that have none."""
    insts = [_rows_of(60, 8, [3], 1), _rows_of(64, 70, [3, 4], 2), _rows_of(200, 4, [2, 3], 3), _rows_of(45, 40, [3], 4)]
    models = [q.Model("pubo", off=t[0], ids=t[1], coef=t[2]) for t in insts]
    params = {"seed": 6, "sweeps": 12, "restarts": 9, "beta_start": 0.05, "beta_stop": 2.0, "rng_mode": mode}
    b = q.Batch(models, SA, {"params": params}).run()
    for i, m in enumerate(models):
        plain = q.Solver(m, SA, {"params": dict(params, kernel="warp")}).init().run().result()
        assert b.result(i)["solutions"] == plain["solutions"], i
