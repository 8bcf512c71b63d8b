"""Quantum Monte Carlo with few decisions a launch: the kernel of many launches and of
one gives the same slices (GPU required)."""
import numpy as np
import pytest

import qiotoolkit_gb300 as q
from qiotoolkit_gb300 import instances as I

pytestmark = pytest.mark.gpu

KEYS = ("cost", "lowest", "attempts", "accepts", "states", "lowest_states")


# launches of fewer decisions than a 64th of the variables; a cost limit ends each after one sweep
@pytest.mark.parametrize("sweeps", [5, 6, 7, 60])
def test_qmc_few_decisions(sweeps):
    off, ids, coef = I.weighted_maxsat(400, seed=3)
    m = q.Model("maxsat", off=off, ids=ids, coef=coef)
    n = m.n_vars // 64
    assert 5 <= n <= 6
    params = {"seed": 3, "sweeps": sweeps, "restarts": 3, "trotter_number": 12, "beta_start": 0.5, "beta_stop": 3.0,
              "transverse_field_low": 0.0, "transverse_field_high": 2.0}
    g = q.Solver(m, "quantummontecarlo.qiotoolkit", {"params": params}).init().run().replicas()
    h = q.Solver(m, "quantummontecarlo.qiotoolkit", {"params": dict(params, cost_limit=-1e300)}).init().run().replicas()
    for key in KEYS:
        np.testing.assert_array_equal(g[key], h[key], err_msg=key)
