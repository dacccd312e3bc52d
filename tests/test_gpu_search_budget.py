"""A time budget of the batched search holds to within a batch, also where the
search has come to evaluate many batches in one launch: at a local optimum of
the full-scale pair no batch accepts anything, and a whole pass could be one."""
import numpy as np
import pytest

import bmb200 as bm
from conftest import make_engine

pytestmark = pytest.mark.gpu


def test_budget_holds():
    A, B, _, init = bm.gen_pair(2)
    e = make_engine(A.n, (A.src, A.dst, A.w), (B.src, B.dst, B.w), init)
    rows = bm.rows_from_ordering(bm.ordering_by_weighted_degree(A))
    e.search_batched(rows)
    e.set_path("gain_tables", -1)
    p, _ = e.search_batched(rows, rows_per_batch=64)
    assert p.converged and p.sweeps == 1
    whole = p.seconds
    assert whole > 2e-3
    # what a launch of one batch can take: a few hundred microseconds with the
    # host's part and its noise (the least of five runs is taken), while half a
    # pass in one launch takes milliseconds
    over = []
    for budget in np.linspace(0.15, 0.8, 14) * whole:
        runs = []
        for _ in range(5):
            p, st = e.search_batched(rows, rows_per_batch=64, time_budget=float(budget))
            if not p.converged:
                assert p.rows_done % 64 == 0 and p.rows_done < A.n
            runs.append(p.seconds - budget)
        over.append(min(runs))
    assert max(over) < 0.1 * whole, (whole, over)
    e.close()
