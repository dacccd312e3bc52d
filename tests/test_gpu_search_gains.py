"""The batched search with gain tables and batches evaluated ahead against the
same search a pass a call (which keeps no tables and starts each pass with
single batches): the same mapping, score and accepts, exactly."""
import numpy as np
import pytest

import bmb200 as bm
from conftest import golden_graphs, make_engine
from oracle_bind import Oracle

pytestmark = pytest.mark.gpu


def _both(n, A, B, pi, R, rows=None, passes=60):
    e, f = make_engine(n, A, B, pi), make_engine(n, A, B, pi)
    p, _ = e.search_batched(rows, rows_per_batch=R, max_sweeps=passes)
    q = bm.Progress()
    while not q.converged and q.sweeps < passes:
        q, _ = f.search_batched(rows, rows_per_batch=R, max_sweeps=q.sweeps + 1, prog=q)
    np.testing.assert_array_equal(e.get_mapping(), f.get_mapping())
    for name in ("rows_done", "evaluated", "accepts", "score", "launches", "sweeps", "converged", "next_row_pos"):
        assert getattr(p, name) == getattr(q, name), name
    np.testing.assert_array_equal(e.overlap(), f.overlap())
    # the lists that later calls read are those of the final mapping
    check = np.arange(1, min(n, 40) + 1, dtype=np.int32)
    np.testing.assert_array_equal(e.delta_rows(check), f.delta_rows(check))
    score = e.score()
    e.close()
    f.close()
    return score


@pytest.mark.parametrize("n,m,deg,R", [(5, 12, 4, 2), (300, 4000, 80, 7), (301, 9000, 200, 300), (2000, 40_000, 500, 64),
                                       (3003, 200_000, 2000, 296)])
def test_equals_a_pass_a_call(n, m, deg, R):
    A, B, _, init = bm.gen_pair(1 if n < 2500 else 3, n=n, m_target=m, max_degree=deg, seed=n, init_mode=int(n == 2000))
    GA, GB = (A.src, A.dst, A.w), (B.src, B.dst, B.w)
    rows = (np.random.default_rng(n).permutation(n) + 1).astype(np.int32)
    score = _both(n, GA, GB, init, R, rows)
    assert score >= Oracle(n, GA, GB).score(init)


@pytest.mark.parametrize("name", ["golden_selfloop_ref", "golden_selfloop"])
def test_selfloops_and_repeats(request, name):
    g = request.getfixturevalue(name)
    n, A, B = golden_graphs(g)
    _both(n, A, B, g["pi_init"] if "pi_init" in g else g["pis"][0], 16)


def test_budgets_stop_between_batches(golden_cfg1):
    n, A, B = golden_graphs(golden_cfg1)
    for budget in (dict(max_accepts=900), dict(target_score=90_000)):
        e, f = (make_engine(n, A, B, golden_cfg1["pi_init"]) for _ in range(2))
        p, _ = e.search_batched(rows_per_batch=64, **budget)
        q = bm.Progress()
        while True:  # one batch a call at most, by a budget of one accept
            left = budget["max_accepts"] - q.accepts if "max_accepts" in budget else 1 << 30
            if left <= 0 or q.converged or f.tracked_score() >= budget.get("target_score", 1 << 60):
                break
            q, _ = f.search_batched(rows_per_batch=64, max_accepts=1, prog=q)
        assert (p.accepts, p.score) == (q.accepts, q.score)
        np.testing.assert_array_equal(e.get_mapping(), f.get_mapping())
        e.close()
        f.close()
