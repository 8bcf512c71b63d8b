"""Costs and cost differences of given states against the oracle, bit for bit
(GPU required): FP64 sums in term order where their running value changes its
binade, meets ties or cancels, state rows of odd widths and any nonzero byte."""
import numpy as np
import pytest

import qiotoolkit_gb300 as q
from oracle import oracle as O

pytestmark = pytest.mark.gpu

COEFS = {
    "normal": lambda rng, n: rng.standard_normal(n),
    "wide": lambda rng, n: rng.standard_normal(n) * 10.0 ** rng.integers(-18, 19, n),
    "extreme": lambda rng, n: rng.choice([1e300, -1e300, 1e-300, 5e-324, 1.0, -3.5], n),
    "ties": lambda rng, n: rng.choice([2.0**52, -(2.0**52), 2.0**53 + 2, 0.5, -0.5, 1.5, 1.0], n),
    "powers": lambda rng, n: rng.choice([1.0, -1.0], n) * 2.0 ** rng.integers(-3, 60, n),
    "cancel": lambda rng, n: np.repeat(rng.standard_normal((n + 1) // 2), 2)[:n] * np.resize([1.0, -1.0], n),
}


@pytest.mark.parametrize("kind", ["ising", "pubo"])
@pytest.mark.parametrize("coefs", list(COEFS))
@pytest.mark.parametrize("n", [3, 32, 77, 200])
def test_state_costs(kind, coefs, n):
    rng = np.random.default_rng(n)
    rows = sorted({tuple(sorted(rng.choice(n, int(rng.integers(1, min(n, 4) + 1)), replace=False).tolist()))
                   for _ in range(6 * n)} | {(v,) for v in range(n)})
    rng.shuffle(rows)
    c = COEFS[coefs](rng, len(rows))
    inst = O.flatten_terms([(float(x), list(t)) for x, t in zip(c, rows)])
    at = dict(zip(("off", "ids", "coef"), inst))
    g, o = q.Model(kind, **at), O.Model(kind, **at)
    states = rng.integers(0, 2, (67, n), dtype=np.uint8)
    marked = states * rng.integers(1, 256, states.shape).astype(np.uint8)  # any nonzero byte
    np.testing.assert_array_equal(g.calculate_cost(marked), [o.cost(s) for s in states])
    v = rng.integers(0, n, len(states))
    np.testing.assert_array_equal(g.calculate_cost_difference(marked, v),
                                  [o.cost_difference(s, int(x)) for s, x in zip(states, v)])


@pytest.mark.parametrize("n_states", [1, 31, 32, 33, 127, 128, 129])
def test_few_states(n_states):
    """Around 2 KB (costs) and 8 KB (differences) of 64 variables' state bytes, from
    where the device packs them."""
    rng = np.random.default_rng(n_states)
    rows = [[v] for v in range(64)] + [sorted(rng.choice(64, 3, replace=False).tolist()) for _ in range(100)]
    at = dict(zip(("off", "ids", "coef"), O.flatten_terms([(float(x), r) for x, r in zip(rng.standard_normal(164), rows)])))
    g, o = q.Model("pubo", **at), O.Model("pubo", **at)
    states = rng.integers(0, 2, (n_states, 64), dtype=np.uint8)
    marked = states * rng.integers(1, 256, states.shape).astype(np.uint8)
    np.testing.assert_array_equal(g.calculate_cost(marked), [o.cost(s) for s in states])
    v = rng.integers(0, 64, n_states)
    np.testing.assert_array_equal(g.calculate_cost_difference(marked, v),
                                  [o.cost_difference(s, int(x)) for s, x in zip(states, v)])
