"""Best permutations found by the assignment table (calls without
per-permutation output) against the enumeration of every permutation, which
the tests of the permutation sets hold against the oracle."""
import itertools

import numpy as np
import pytest

import bmb200 as bm
from conftest import golden_graphs, make_engine

pytestmark = pytest.mark.gpu


def _check(e, k, sets):
    best, perm = e.kset_eval(k, sets)
    b2, p2, alld = e.kset_eval(k, sets, all_deltas=True)
    first = alld.argmax(axis=1)  # the first maximum in lexicographic order
    np.testing.assert_array_equal(best, alld[np.arange(len(sets)), first])
    perms = np.array(list(itertools.permutations(range(k))), np.int32)
    np.testing.assert_array_equal(perm, perms[first])
    np.testing.assert_array_equal(best, b2)
    np.testing.assert_array_equal(perm, p2)


def _sets(A, n, k, count, rng):
    """Random sets, and sets grown around edges (2 to k members with internal entries)."""
    out = [rng.choice(n, k, replace=False) + 1 for _ in range(count)]
    src, dst = np.asarray(A[0]), np.asarray(A[1])
    for i in range(count):
        inside = []
        while len(inside) < 2 + i % (k - 1):
            e = int(rng.integers(len(src)))
            for v in (int(src[e]), int(dst[e])):
                if v not in inside:
                    inside.append(v)
        inside = inside[:k]
        while len(inside) < k:
            v = int(rng.integers(1, n + 1))
            if v not in inside:
                inside.append(v)
        out.append(rng.permutation(inside))
    return np.array(out, np.int32)


@pytest.mark.parametrize("k", [2, 3, 4, 5, 6, 7, 8])
def test_random_and_connected_sets(golden_cfg1, k):
    n, A, B = golden_graphs(golden_cfg1)
    e = make_engine(n, A, B, golden_cfg1["pi_init"])
    _check(e, k, _sets(A, n, k, 12, np.random.default_rng(k)))
    e.close()


@pytest.mark.parametrize("k", [4, 8])
def test_selfloops_and_repeated_edges(golden_selfloop, golden_selfloop_ref, k):
    n, A, B = golden_graphs(golden_selfloop_ref)
    e = make_engine(n, A, B, golden_selfloop_ref["pi_init"])
    _check(e, k, _sets(A, n, k, 8, np.random.default_rng(20 + k)))
    e.close()
    n, A, B = golden_graphs(golden_selfloop)
    e = make_engine(n, A, B, golden_selfloop["pis"][0])
    _check(e, min(k, n), _sets(A, n, min(k, n), 4, np.random.default_rng(30 + k)))
    e.close()


def test_ties_take_the_first_permutation():
    # unit weights on a sparse pair: most totals tie
    n = 64
    rng = np.random.default_rng(3)
    src, dst = rng.integers(1, n + 1, (2, 200)).astype(np.int32)
    key = np.unique(src.astype(np.int64) * 1000 + dst)
    src, dst = (key // 1000).astype(np.int32), (key % 1000).astype(np.int32)
    keep = src != dst
    G = (src[keep], dst[keep], np.ones(keep.sum(), np.int32))
    e = make_engine(n, G, G, np.concatenate([[0], rng.permutation(n) + 1]))
    for k in (4, 6, 8):
        _check(e, k, _sets(G, n, k, 16, rng))
    e.close()


def test_hub_rows_past_the_staging_and_large_ids():
    A, B, _, init = bm.gen_pair(3, n=2000, m_target=160_000, max_degree=1900, seed=5)
    deg = np.bincount(A.src, minlength=A.n + 1) + np.bincount(A.dst, minlength=A.n + 1)
    hubs = np.argsort(-deg)[:16].astype(np.int32)
    e = make_engine(A.n, (A.src, A.dst, A.w), (B.src, B.dst, B.w), init)
    _check(e, 8, hubs.reshape(2, 8))
    e.close()
    n = 131071  # bitmaps past the default shared-memory limit
    rng = np.random.default_rng(9)
    src, dst = rng.integers(n - 300, n + 1, (2, 3000)).astype(np.int32)
    key = np.unique(src.astype(np.int64) * 200_000 + dst)
    src, dst = (key // 200_000).astype(np.int32), (key % 200_000).astype(np.int32)
    keep = src != dst
    G = (src[keep], dst[keep], rng.integers(1, 9, keep.sum()).astype(np.int32))
    pi = np.arange(n + 1)
    pi[n - 300:] = rng.permutation(pi[n - 300:])
    e = make_engine(n, G, G, pi)
    _check(e, 5, (rng.permutation(300)[:40] + n - 299).reshape(8, 5).astype(np.int32))
    e.close()
