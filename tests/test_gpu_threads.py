"""Solves of different sizes on several threads at once (GPU required).  Their
kernels' shared memory differs, and the limit that a launch needs belongs to the
kernel, not to the thread: no launch may be refused, and every solve returns what
it returns alone."""
import threading

import numpy as np
import pytest

import qiotoolkit_gb300 as q
from qiotoolkit_gb300 import instances as I

pytestmark = pytest.mark.gpu

QMC = {"trotter_number": 4, "beta_start": 1.0, "beta_stop": 5.0, "transverse_field_low": 0.0,
       "transverse_field_high": 3.0}


# sizes of which each takes another amount of shared memory above the default limit
@pytest.mark.parametrize("target,sizes,extra", [("tabu.qiotoolkit", (1184, 1500, 2200, 3300), {"tabu_tenure": 9}),
                                                ("quantummontecarlo.qiotoolkit", (4200, 6000, 9000, 16000), QMC),
                                                ("simulatedannealing.qiotoolkit", (3000, 8000, 16000, 30000),
                                                 {"kernel": "warp"})])
def test_threads_of_different_sizes(target, sizes, extra):
    # (a limit that is never reached: a launch a step)
    params = dict(extra, seed=5, sweeps=100, restarts=2, cost_limit=-1e300)
    models = []
    for n in sizes:
        off, ids, coef = I.er_ising_gauss(n, 4, seed=n)
        models.append(q.Model("ising", off=off, ids=ids, coef=coef))

    def solve(m):
        return q.Solver(m, target, {"params": params}).init().run().replicas()

    alone = [solve(m) for m in models]
    got, failed = [None] * len(models), []

    def work(i):
        try:
            got[i] = solve(models[i])
        except Exception as e:
            failed.append(f"{sizes[i]} variables: {e}")

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(models))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
    for a, b in zip(alone, got):
        for key in a:
            np.testing.assert_array_equal(a[key], b[key], err_msg=key)
