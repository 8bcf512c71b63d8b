"""Tabu search around its scan's 128 variables and around the models that live in
shared memory (their rows decide), rows of more than 32 terms, against the oracle,
bit for bit (GPU required): sweeps in one launch and in launches of one."""
import numpy as np
import pytest

import qiotoolkit_gb300 as q
from qiotoolkit_gb300 import instances as I
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [None, -1e300])
@pytest.mark.parametrize("n,edges,integer", [(31, 90, False), (128, 384, True), (129, 5000, False), (1184, 3552, False),
                                             (2900, 8700, False), (3300, 9900, False), (3300, 9900, True)])
def test_tabu_sizes(n, edges, integer, limit):
    off, ids, coef = I.er_ising(n, edges, seed=n)
    coef = np.sign(coef) if integer else coef
    inst = {"off": off, "ids": ids, "coef": coef}
    params = {"seed": 5, "sweeps": 60, "restarts": 6, "tabu_tenure": 9}
    if limit is not None:
        params["cost_limit"] = limit
    s = q.Solver(q.Model("ising", **inst), "tabu.qiotoolkit", {"params": params}).init().run()
    r = O.run(O.Model("ising", **inst), "tabu", seed=5, step_limit=60, restarts=6, tabu_tenure=9)
    g = s.replicas()
    for key in ("cost", "lowest", "attempts", "accepts", "states", "lowest_states"):
        np.testing.assert_array_equal(g[key], getattr(r, key), err_msg=key)
