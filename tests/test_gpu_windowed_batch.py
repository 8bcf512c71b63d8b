"""Windowed kernel, batch queue: Ising models of terms of up to seven members, whose
flips mark different numbers of later incidences on the warp's lanes, against the
same models' plain solves (GPU required)."""
import numpy as np
import pytest

import qiotoolkit_gb300 as q
from qiotoolkit_gb300 import instances as I

pytestmark = pytest.mark.gpu

SA = "simulatedannealing.qiotoolkit"


def _models(kind, count, seed):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(count):
        n = int(rng.integers(16, 65))
        ids = {tuple(sorted(rng.choice(n, int(rng.integers(1, 8)), replace=False).tolist()))
               for _ in range(int(n * rng.uniform(1, 4)))}
        ids = [list(t) for t in sorted(ids, key=lambda t: rng.random())]
        coef = rng.choice([-1.0, 1.0], len(ids)) if rng.random() < 0.5 else rng.standard_normal(len(ids))
        off, flat, coef = I._pack(ids, coef)
        out.append(q.Model(kind, off=off, ids=flat, coef=coef))
    return out


@pytest.mark.parametrize("kind", ["ising", "pubo"])
@pytest.mark.parametrize("mode", ["replay", "counter"])
def test_windowed_batches_equal_plain_solves(kind, mode):
    models = _models(kind, 300, 7)
    params = {"seed": 5, "sweeps": 24, "restarts": 6, "beta_start": 0.3, "beta_stop": 2.0, "rng_mode": mode,
              "number_of_solutions": 6, "kernel": "warp"}
    b = q.Batch(models, SA, {"params": params}).run()
    for i, m in enumerate(models):
        assert b.result(i)["solutions"] == q.Solver(m, SA, {"params": params}).init().run().result()["solutions"], i
