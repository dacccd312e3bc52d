"""The auction at its edges: bidder counts around the groups of warps, ties,
values that need 64 bits from the start, and values whose prices outgrow 32
bits on the way, against scipy's optimal assignment."""
import numpy as np
import pytest
from scipy.optimize import linear_sum_assignment

import bmb200 as bm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 2, 3, 15, 16, 17, 31, 32, 33, 65, 1023, 1025, 2049])
@pytest.mark.parametrize("kind", ["ties", "sparse", "wide", "outgrow", "negative"])
def test_optimal_totals(k, kind):
    rng = np.random.default_rng(k)
    a = rng.integers(0, 3, (k, k))
    if kind == "sparse":  # few objects are worth anything: long chains of single bidders
        a = np.where(rng.random((k, k)) < 0.02, rng.integers(1, 2000, (k, k)), 0)
    elif kind == "wide":
        a = rng.integers(-(1 << 30), (1 << 30) + 1, (k, k))
        a[0, 0] = 1 << 30
    elif kind == "outgrow":  # k + 1 times the largest is just below 2^30
        top = ((1 << 30) - 1) // (k + 1)
        a = rng.integers(0, 2, (k, k)) * top
        a[:, 0] = top
    elif kind == "negative":
        a = -rng.integers(0, 500, (k, k))
    a = np.ascontiguousarray(a, np.int32)
    with bm.Engine(0) as e:
        assign, total = e.lap_solve(a)
    assert sorted(assign.tolist()) == list(range(k))
    assert total == int(a[np.arange(k), assign].astype(np.int64).sum())
    if k <= 1100 or kind in ("sparse", "wide"):
        r, c = linear_sum_assignment(a, maximize=True)
        assert total == int(a[r, c].astype(np.int64).sum())
