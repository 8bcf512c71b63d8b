"""Initial states and costs (GPU required) at the edges of the initialising
kernel's two forms, a warp and a block to a walker: 512 terms, and from there 2048
walkers (FP64) or 8192 (integers); walkers that do not fill a block.  Against the
oracle, bit for bit."""
import numpy as np
import pytest

import qiotoolkit_gb300 as q
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _terms(n, count, kind, integer, seed):
    rng = np.random.default_rng(seed)
    rows = [[v] for v in range(n)]
    while len(rows) < count:
        rows.append(sorted(rng.choice(n, int(rng.integers(2, 4)), replace=False).tolist()))
    rows = {tuple(r): None for r in rows}
    while len(rows) < count:
        rows[tuple(sorted(rng.choice(n, 3, replace=False).tolist()))] = None
    c = rng.choice([-2.0, -1.0, 1.0, 3.0], count) if integer else rng.standard_normal(count)
    rows = [[v + 1 for v in r] for r in rows]
    if kind == "maxsat":
        rows = [[int(v * rng.choice([-1, 1])) for v in r] for r in rows]
        c = np.abs(c)
    return O.flatten_terms([(float(x), r) for x, r in zip(c, rows)])


@pytest.mark.parametrize("mode", ["replay", "counter"])
@pytest.mark.parametrize("kind,count,walkers,integer", [
    ("ising", 100, 1, False), ("pubo", 100, 5, False), ("maxsat", 130, 7, False), ("ising", 512, 6, True),
    ("pubo", 513, 2047, False), ("pubo", 513, 2049, False), ("maxsat", 600, 2048, False), ("maxsat", 600, 3, True),
    ("ising", 513, 8191, True), ("ising", 513, 8194, True), ("ising_plain", 700, 9, False)])
def test_initial_states(kind, count, walkers, integer, mode):
    off, ids, coef = _terms(90, count, kind, integer, count)
    params = {"seed": 11, "sweeps": 2, "restarts": walkers, "beta_start": 0.5, "beta_stop": 2.0, "rng_mode": mode,
              "maxsat_full_sweep": True}
    m = q.Model(kind, off=off, ids=ids, coef=coef)
    s = q.Solver(m, "simulatedannealing.qiotoolkit", {"params": params}).init()
    got = s.replicas()
    np.testing.assert_array_equal(got["cost"], got["lowest"])
    np.testing.assert_array_equal(got["states"], got["lowest_states"])
    o = O.Model(kind, off=off, ids=ids, coef=coef)
    for i in sorted({0, 1, walkers // 2, walkers - 1} & set(range(walkers))):
        assert got["cost"][i] == o.cost(got["states"][i])
    if walkers < 100:
        r = O.run(o, "sa", seed=11, step_limit=2, restarts=walkers, sched=("linear", 0.5, 2.0), rng_mode=mode,
                  full_maxsat_sweep=True)
        g = s.run().replicas()
        for key in ("cost", "lowest", "states", "lowest_states"):
            np.testing.assert_array_equal(g[key], getattr(r, key), err_msg=key)
