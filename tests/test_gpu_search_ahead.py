"""Batches evaluated ahead, at the most rows that a launch of several batches
holds (20,000), against the same batches one call each: best partners, the
independent subset, the swaps applied."""
import numpy as np
import pytest

import bmb200 as bm
from conftest import make_engine

pytestmark = pytest.mark.gpu


def _stepwise(e, rows, R, passes):
    accepts = 0
    for _ in range(passes):
        for at in range(0, len(rows), R):
            r = e.rows_best(rows[at:at + R])
            r = r[r["best_delta"] > 0]
            pairs = np.stack([r["row"], r["best"]], 1).astype(np.int32)
            chosen = e.select_independent(pairs, r["best_delta"])
            if len(chosen):
                e.apply_swaps(pairs[chosen], r["best_delta"][chosen])
            accepts += len(chosen)
    return accepts


@pytest.mark.parametrize("n,R", [(20_000, 2999), (20_000, 3000), (24_000, 400), (24_000, 6000), (24_000, 7001),
                                 (24_000, 20_000), (24_000, 22_000), (24_000, 24_000)])
def test_equals_batch_by_batch(n, R):
    # few vertices have edges, so that most batches accept nothing and launches grow
    A, B, _, init = bm.gen_pair(1, n=400, m_target=5000, max_degree=90, seed=R, init_mode=0)
    rng = np.random.default_rng(R)
    at = np.concatenate([[0], 1 + rng.permutation(n)[:400]]).astype(np.int32)
    GA, GB = ((at[g.src], at[g.dst], g.w) for g in (A, B))
    pi = np.concatenate([[0], rng.permutation(n) + 1]).astype(np.int32)
    # the vertices with edges, and at whose images B has some, come first
    busy = np.isin(np.arange(1, n + 1), at[1:]) | np.isin(pi[1:], at[1:])
    rows = (np.argsort(~busy, kind="stable") + 1).astype(np.int32)
    e, f = make_engine(n, GA, GB, pi), make_engine(n, GA, GB, pi)
    p, _ = e.search_batched(rows, rows_per_batch=R, max_sweeps=3)
    accepts = _stepwise(f, rows, R, p.sweeps)
    assert p.accepts == accepts > 0
    assert p.rows_done == p.sweeps * n and p.launches == p.sweeps * -(-n // R)
    np.testing.assert_array_equal(e.get_mapping(), f.get_mapping())
    assert p.score == e.score() == f.score()
    e.close()
    f.close()
