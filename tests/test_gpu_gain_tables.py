"""The batched search reading its batches from the gain tables (forced from the
first batch on) against the same search without them: tables filled from the
rows, updated by every swap of the search, and read for every batch, so a wrong
entry anywhere changes a swap, the mapping or the score."""
import numpy as np
import pytest

import bmb200 as bm
from conftest import golden_graphs, make_engine

pytestmark = pytest.mark.gpu

FIELDS = ("rows_done", "evaluated", "accepts", "score", "launches", "sweeps", "converged", "next_row_pos")


def _compare(n, A, B, pi, R, passes, rows=None, semantics="exact", possible=True):
    """Both searches; returns the accepts."""
    out = []
    for mode in (1, -1):
        e = make_engine(n, A, B, pi)
        e.set_semantics(semantics)
        e.set_path("gain_tables", mode)
        assert e.path("gain_tables") == mode
        before = e.launch_count()
        p, _ = e.search_batched(rows, rows_per_batch=R, max_sweeps=passes)
        check = np.arange(1, min(n, 40) + 1, dtype=np.int32)
        out.append((p, e.get_mapping(), e.overlap(), e.delta_rows(check), e.launch_count() - before))
        assert e.score() == p.score
        e.close()
    (p, *got, used), (q, *want, plain) = out
    for name in FIELDS:
        assert getattr(p, name) == getattr(q, name), name
    for x, y in zip(got, want):
        np.testing.assert_array_equal(x, y)
    assert (used != plain) == possible  # filling and updating the tables are launches of their own
    return p.accepts


# the smallest; columns past the last group of four; batches of a few rows and of
# whole passes, whose first ones accept more swaps than the lists hold at once (64)
@pytest.mark.parametrize("n,m,deg,R,passes", [
    (3, 4, 2, 3, 20), (4, 8, 3, 1, 20), (5, 12, 4, 2, 20), (31, 200, 20, 8, 20), (300, 4000, 80, 7, 20),
    (301, 9000, 200, 300, 30), (2000, 40_000, 500, 64, 12), (2001, 30_000, 400, 2001, 12), (3002, 200_000, 2000, 296, 12),
    (3003, 60_000, 1500, 3003, 12)])
def test_equals_scattered_rows(n, m, deg, R, passes):
    A, B, _, _ = bm.gen_pair(1 if n < 2500 else 3, n=n, m_target=m, max_degree=deg, seed=n)
    rng = np.random.default_rng(n)
    pi = np.concatenate([[0], rng.permutation(n) + 1]).astype(np.int32)  # far from an optimum: many swaps
    rows = (rng.permutation(n) + 1).astype(np.int32)
    accepts = _compare(n, (A.src, A.dst, A.w), (B.src, B.dst, B.w), pi, R, passes, rows)
    assert accepts > (64 if R >= 2000 else 0) or n < 10


def test_more_ids_than_one_range_of_marks():
    n = 20_011  # the lists of a swap are marked 16,384 ids at a time
    A, B, _, init = bm.gen_pair(3, n=n, m_target=10 * n, max_degree=6000, seed=5)
    assert _compare(n, (A.src, A.dst, A.w), (B.src, B.dst, B.w), init, 1000, 2) > 64


def test_some_rows_only():
    n = 1500
    A, B, _, init = bm.gen_pair(3, n=n, m_target=60_000, max_degree=900, seed=6)
    rows = (np.random.default_rng(6).permutation(n)[:100] + 1).astype(np.int32)
    assert _compare(n, (A.src, A.dst, A.w), (B.src, B.dst, B.w), init, 16, 10, rows) > 0


def _loops(n, m, rng, repeats):
    src, dst = rng.integers(1, n + 1, (2, m)).astype(np.int32)
    keep = src != dst
    key = src[keep].astype(np.int64) * (n + 1) + dst[keep]
    _, first = np.unique(key, return_index=True)  # each edge once
    src, dst = src[keep][first], dst[keep][first]
    loops = rng.permutation(n)[:n // 3].astype(np.int32) + 1
    if repeats:
        src, dst = np.concatenate([src, src[:50]]), np.concatenate([dst, dst[:50]])
    src, dst = np.concatenate([src, loops]), np.concatenate([dst, loops])
    return src, dst, rng.integers(1, 200, len(src)).astype(np.int32)


@pytest.mark.parametrize("semantics,repeats,possible", [("exact", False, True), ("exact", True, False),
                                                        ("ref-cpu", False, False)])
def test_selfloops_and_repeated_edges(semantics, repeats, possible):
    n, rng = 700, np.random.default_rng(8)
    A, B = _loops(n, 20_000, rng, repeats), _loops(n, 20_000, rng, True)
    pi = np.concatenate([[0], rng.permutation(n) + 1]).astype(np.int32)
    assert _compare(n, A, B, pi, 50, 8, semantics=semantics, possible=possible) > 64


def test_reference_deltas_without_selfloops():
    n, rng = 600, np.random.default_rng(9)
    A, B = (bm.gen_pair(1, n=n, m_target=9000, max_degree=150, seed=9))[:2]
    pi = np.concatenate([[0], rng.permutation(n) + 1]).astype(np.int32)
    assert _compare(n, (A.src, A.dst, A.w), (B.src, B.dst, B.w), pi, 64, 8, semantics="ref-cpu") > 64


def test_setting_is_checked():
    with bm.Engine(0) as e:
        for path, mode in ((-1, 0), (99, 0), (0, 2), (0, -2)):
            assert e.L.bm_set_path(e.h, path, mode) == bm.BM_INVALID_ARG
        assert e.path("gain_tables") == 0
