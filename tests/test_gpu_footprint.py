"""Device memory at its limits (GPU required), which QIO_DEVICE_MEMORY_LIMIT sets.
Child processes: no other buffers count against the cap.

* The server's footprint of a request covers what its solve holds: a solve whose
  footprint is all that is left runs.  Models with a hub in every block of 32
  variables have the largest tables for their size.
* Costs of given states need no more than the model, the states' spin words and
  the results."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import sys
import numpy as np
import qiotoolkit_gb300 as q
from qiotoolkit_gb300 import instances as I
kind, order = sys.argv[1], int(sys.argv[2])
n = 2048
rng = np.random.default_rng(5)
ids = [[v] for v in range(n)]
for hub in range(0, n, 32):
    for _ in range(180):
        ids.append([hub] + rng.choice(np.setdiff1d(np.arange(n), [hub]), order - 1, replace=False).tolist())
off, ids, coef = I._pack(ids, rng.standard_normal(len(ids)))
m = q.Model(kind, off=off, ids=ids, coef=coef)
srv = q.Server()
rid = srv.submit(m, "simulatedannealing.qiotoolkit", {"seed": 1, "sweeps": 3, "restarts": 2, "beta_start": 0.1, "beta_stop": 2.0})
print(srv.request_bytes(rid), srv.wait(rid)["solutions"]["cost"])
"""


@pytest.mark.parametrize("kind,order", [("ising", 2), ("ising", 3), ("pubo", 2)])
def test_footprint_covers_the_solve(kind, order):
    def run(limit):
        env = dict(os.environ)
        env.pop("QIO_DEVICE_MEMORY_LIMIT", None)
        if limit:
            env["QIO_DEVICE_MEMORY_LIMIT"] = str(limit)
        r = subprocess.run([sys.executable, "-c", CHILD, kind, str(order)], cwd=ROOT, env=env, capture_output=True,
                           text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        size, cost = r.stdout.split()
        return int(size), cost

    size, cost = run(0)
    assert run(size) == (size, cost)


STATES = r"""
import os, sys
import numpy as np
import qiotoolkit_gb300 as q
from qiotoolkit_gb300 import instances as I
off, ids, coef = I.random_pubo(700, 2100, seed=3)
m = q.Model("pubo", off=off, ids=ids, coef=coef)
n, nv = 500, m.n_vars
s = np.random.default_rng(1).integers(0, 2, (n, nv), dtype=np.uint8) * 3
v = np.random.default_rng(2).integers(0, nv, n)
if len(sys.argv) > 1:
    words = (n * ((nv + 31) // 32) * 4 + 255) // 256 * 256
    out = n * 16 + (-n * 16) % 256
    os.environ["QIO_DEVICE_MEMORY_LIMIT"] = str(m.info.device_bytes + words + out)
print(m.calculate_cost(s).tobytes().hex(), m.calculate_cost_difference(s, v).tobytes().hex())
"""


def test_state_costs_without_room_for_bytes():
    def run(*args):
        env = {k: v for k, v in os.environ.items() if k != "QIO_DEVICE_MEMORY_LIMIT"}
        r = subprocess.run([sys.executable, "-c", STATES, *args], cwd=ROOT, env=env, capture_output=True, text=True,
                           timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        return r.stdout

    assert run("capped") == run()
