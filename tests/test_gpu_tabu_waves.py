"""Tabu search with walkers on both sides of one wave of the kernel in shared memory,
against the oracle, bit for bit (GPU required)."""
import numpy as np
import pytest

import qiotoolkit_gb300 as q
from qiotoolkit_gb300 import instances as I
from oracle import oracle as O

pytestmark = pytest.mark.gpu

KEYS = ("cost", "lowest", "attempts", "accepts", "states", "lowest_states")


# 152 walkers are one wave of the kernel in shared memory, which holds one a block
@pytest.mark.parametrize("n,edges,restarts", [(3000, 4500, 152), (3000, 4500, 153), (1000, 8000, 153)])
def test_tabu_waves(n, edges, restarts):
    off, ids, coef = I.er_ising(n, edges, seed=n)
    inst = {"off": off, "ids": ids, "coef": coef}
    s = q.Solver(q.Model("ising", **inst), "tabu.qiotoolkit",
                 {"params": {"seed": 5, "sweeps": 8, "restarts": restarts, "tabu_tenure": 9}}).init().run()
    r = O.run(O.Model("ising", **inst), "tabu", seed=5, step_limit=8, restarts=restarts, tabu_tenure=9)
    g = s.replicas()
    for key in KEYS:
        np.testing.assert_array_equal(g[key], getattr(r, key), err_msg=key)
