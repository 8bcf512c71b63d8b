"""Kernels that "auto" picks on both sides of its lines -- walkers and variables
-- give the same walkers as the kernels asked for by name (GPU
required)."""
import numpy as np
import pytest

import qiotoolkit_gb300 as q
from qiotoolkit_gb300 import instances as I

pytestmark = pytest.mark.gpu

SA = "simulatedannealing.qiotoolkit"
KEYS = ("cost", "lowest", "attempts", "accepts", "states", "lowest_states")


def _same(a, b):
    for key in KEYS:
        np.testing.assert_array_equal(a[key], b[key], err_msg=key)


MODELS = {
    "er32": ("ising", lambda: I.er_ising(32, 64, seed=1)),
    "er33": ("ising", lambda: I.er_ising(33, 66, seed=1)),
    "er64": ("ising", lambda: I.er_ising(64, 192, seed=1)),
    "pubo16": ("pubo", lambda: I.random_pubo(16, 40, seed=1)),
    "pubo64": ("pubo", lambda: I.random_pubo(64, 160, seed=1)),
    "pubo65": ("pubo", lambda: I.random_pubo(65, 160, seed=1)),
    "ising3_40": ("ising", lambda: I.random_pubo(40, 100, seed=1)),
    "sat20": ("maxsat", lambda: I.weighted_maxsat(20, seed=1)),
    "sat64": ("maxsat", lambda: I.weighted_maxsat(64, seed=1)),
}


# one wave of the block-decided sweep, two; the lane kernel's line at 64 spins
@pytest.mark.parametrize("name,walkers", [(n, w) for n in MODELS for w in (608, 609, 1216, 1217)] +
                         [("er64", 10239), ("er64", 10240)])
@pytest.mark.parametrize("mode", ["replay", "counter"])
def test_auto_equals_named_kernels(name, walkers, mode):
    kind, gen = MODELS[name]
    off, ids, coef = gen()
    m = q.Model(kind, off=off, ids=ids, coef=coef)
    params = {"seed": 11, "sweeps": 7, "restarts": walkers, "beta_start": 0.2, "beta_stop": 2.0, "rng_mode": mode}
    if kind == "maxsat":
        params["maxsat_full_sweep"] = True
    auto = q.Solver(m, SA, {"params": params}).init().run()
    g = auto.replicas()
    for kernel in ("fields", "warp"):
        _same(g, q.Solver(m, SA, {"params": dict(params, kernel=kernel)}).init().run().replicas())


def test_batch_of_small_models_equals_named_kernels():
    models = []
    for i in range(40):
        off, ids, coef = I.random_pubo(12 + i, 3 * (12 + i), seed=i)
        models.append(q.Model("pubo", off=off, ids=ids, coef=coef))
    for count in (38, 39, 40):  # 1216 walkers and more
        params = {"seed": 2, "sweeps": 20, "restarts": 32, "beta_start": 0.2, "beta_stop": 2.0}
        out = [q.Batch(models[:count], SA, {"params": dict(params, kernel=k)}).run() for k in ("auto", "fields", "warp")]
        for i in range(count):
            docs = [b.result(i)["solutions"] for b in out]
            assert docs[0] == docs[1] == docs[2]
