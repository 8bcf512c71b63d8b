"""A device without room for the block-decided sweep's tables runs the model on the
windowed sweep, with the same walkers (GPU required).  Child processes: the cap on
device memory (QIO_DEVICE_MEMORY_LIMIT) is a process's."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import os, sys
import numpy as np
import qiotoolkit_gb300 as q
from qiotoolkit_gb300 import instances as I
rng = np.random.default_rng(5)
n = 2048
ids = [[v] for v in range(n)]
for hub in range(0, n, 32):
    ids += [[hub, int(u)] for u in rng.choice(np.setdiff1d(np.arange(n), [hub]), 180, replace=False)]
off, ids, coef = I._pack(ids, rng.standard_normal(len(ids)))
m = q.Model(sys.argv[1], off=off, ids=ids, coef=coef)
if sys.argv[2] == "capped":
    os.environ["QIO_DEVICE_MEMORY_LIMIT"] = str(m.info.device_bytes - 4096)
s = q.Solver(m, sys.argv[3], {"seed": 1, "sweeps": 4, "restarts": 3, "beta_start": 0.1, "beta_stop": 2.0,
                              "temperatures": {"type": "geometric", "initial": 0.5, "final": 3.0, "count": 3}}
             if "tempering" in sys.argv[3] else
             {"seed": 1, "sweeps": 4, "restarts": 3, "beta_start": 0.1, "beta_stop": 2.0}).init().run()
r = s.replicas()
print(s.stats().sweep_kernel, *(r[k].tobytes().hex() for k in ("cost", "lowest", "accepts", "states", "lowest_states")))
"""


@pytest.mark.parametrize("kind", ["ising", "pubo"])
@pytest.mark.parametrize("target", ["simulatedannealing.qiotoolkit", "paralleltempering.qiotoolkit"])
def test_without_room_for_tables(kind, target):
    def run(cap):
        env = {k: v for k, v in os.environ.items() if k != "QIO_DEVICE_MEMORY_LIMIT"}
        r = subprocess.run([sys.executable, "-c", CHILD, kind, cap, target], cwd=ROOT, env=env, capture_output=True,
                           text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        return r.stdout.split(" ", 1)

    kernel, walkers = run("")
    capped, same = run("capped")
    assert (kernel, capped) == ("8", "1") and same == walkers
