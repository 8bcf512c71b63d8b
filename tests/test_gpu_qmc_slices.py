"""Edges of quantum Monte Carlo with a lane per slice against the oracle, bit
for bit (GPU required): one to 32 slices and one more, a single variable, rows
of more than 32 terms, terms of more members than are loaded ahead, negated
literals, sweeps cut into launches of one."""
import itertools

import numpy as np
import pytest

import qiotoolkit_gb300 as q
from oracle import oracle as O

pytestmark = pytest.mark.gpu

QMC = "quantummontecarlo.qiotoolkit"


def instance(n, sizes, count, seed, hub=0, integer=False):
    rng = np.random.default_rng(seed)
    rows = {(v,) for v in range(n)}
    for _ in range(count):
        rows.add(tuple(sorted(rng.choice(n, min(n, int(rng.choice(sizes))), replace=False).tolist())))
    for _ in range(hub):
        rows.add(tuple(sorted({n // 2, *rng.choice(n, 2, replace=False).tolist()})))
    rows = sorted(rows)
    c = rng.choice([-2.0, -1.0, 1.0, 3.0], len(rows)) if integer else rng.normal(size=len(rows))
    return O.flatten_terms([(float(x), list(t)) for x, t in zip(c, rows)])


def signed(seed, **kw):
    off, ids, coef = instance(seed=seed, **kw)
    return off, (np.asarray(ids) + 1) * np.random.default_rng(seed).choice([-1, 1], len(ids)), np.abs(coef)


CASES = {
    "one_variable": ("ising", lambda: instance(1, [1], 0, 1)),
    "pair": ("ising", lambda: instance(65, [2], 200, 2)),
    "pair_hub": ("ising", lambda: instance(150, [2], 200, 3, hub=90, integer=True)),
    "pair_hub_real": ("ising", lambda: instance(150, [2], 200, 3, hub=90)),
    "parity_large": ("ising", lambda: instance(70, [3, 4, 5, 9], 200, 4)),
    "plain": ("ising_plain", lambda: instance(40, [2, 3], 100, 5)),
    "pubo_large": ("pubo", lambda: instance(70, [2, 4, 5, 8], 300, 6, hub=60)),
    "pubo_int": ("pubo", lambda: instance(33, [2, 3, 6], 120, 7, integer=True)),
    "sat": ("maxsat", lambda: signed(8, n=60, sizes=[2, 3, 5], count=250)),
}


@pytest.mark.parametrize("trotter", [3, 31, 32, 33])
@pytest.mark.parametrize("name", list(CASES))
def test_lane_per_slice(name, trotter):
    kind, gen = CASES[name]
    inst = dict(zip(("off", "ids", "coef"), gen()))
    params = {"seed": 5, "sweeps": 15, "restarts": 3, "trotter_number": trotter, "beta_start": 0.5,
              "beta_stop": 4.0, "transverse_field_low": 0.1, "transverse_field_high": 2.0, "maxsat_full_sweep": True,
              "cost_limit": -1e300}
    s = q.Solver(q.Model(kind, **inst), QMC, {"params": params}).init().run()
    r = O.run(O.Model(kind, **inst), "qmc", seed=5, step_limit=15, restarts=3, trotter_number=trotter,
              sched=("linear", 0.5, 4.0), sched2=("linear", 0.1, 2.0), full_maxsat_sweep=True)
    g = s.replicas()
    for key in ("cost", "lowest", "attempts", "accepts", "states", "lowest_states"):
        np.testing.assert_array_equal(g[key], getattr(r, key), err_msg=key)
    assert s.stats().near_ties == 0


def _solve(kind, inst, mode, sweeps, trotter):
    params = {"seed": 5, "sweeps": sweeps, "restarts": 2, "trotter_number": trotter, "beta_start": 0.5, "beta_stop": 4.0,
              "transverse_field_low": 0.1, "transverse_field_high": 2.0, "rng_mode": mode, "kernel": "warp"}
    s = q.Solver(q.Model(kind, **inst), QMC, {"params": params}).init().run()
    r = O.run(O.Model(kind, **inst), "qmc", seed=5, step_limit=sweeps, restarts=2, trotter_number=trotter,
              sched=("linear", 0.5, 4.0), sched2=("linear", 0.1, 2.0), rng_mode=mode)
    g = s.replicas()
    for key in ("cost", "lowest", "attempts", "accepts", "states", "lowest_states"):
        np.testing.assert_array_equal(g[key], getattr(r, key), err_msg=key)


@pytest.mark.parametrize("mode", ["replay", "counter"])
@pytest.mark.parametrize("n,trotter", [(511, 7), (700, 32)])
def test_flip_ring_wraps(n, trotter, mode):
    """Several sweeps in one launch: thousands of flip words through a ring of 512."""
    inst = dict(zip(("off", "ids", "coef"), instance(n, [2], 3 * n, n)))
    _solve("ising", inst, mode, 8, trotter)


@pytest.mark.parametrize("mode", ["replay", "counter"])
@pytest.mark.parametrize("n", [45, 46, 47])
def test_rows_around_the_widest(n, mode):
    """All terms of up to three variables: rows of 991 to 1082 incidences, around the
    widest that a lane per slice takes."""
    rows = [c for k in (1, 2, 3) for c in itertools.combinations(range(n), k)]
    rng = np.random.default_rng(n)
    inst = dict(zip(("off", "ids", "coef"), O.flatten_terms([(float(x), list(t)) for x, t in
                                                             zip(rng.normal(size=len(rows)), rows)])))
    _solve("pubo", inst, mode, 3, 5)
