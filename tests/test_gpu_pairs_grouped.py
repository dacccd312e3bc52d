"""Pair deltas grouped by u (long lists) against the oracle and against the
ungrouped kernel, which shorter lists take, and that kernel at the list
lengths where its share of pairs per block changes."""
import numpy as np
import pytest

import bmb200 as bm
from conftest import golden_graphs, make_engine
from oracle_bind import Oracle

pytestmark = pytest.mark.gpu


def _slices(e, pairs):
    """The same pairs in lists short enough for the ungrouped kernel."""
    step = 1000
    return np.concatenate([e.delta_pairs(pairs[i:i + step]) for i in range(0, len(pairs), step)])


def _lists(n, rng):
    k = (64 if n < 1000 else 10) * n + 37
    rand = rng.integers(1, n + 1, (k, 2)).astype(np.int32)
    one_u = rand.copy()
    one_u[:, 0] = n  # every pair in one group: several items of 256 pairs and a remainder
    runs = rand.copy()
    runs[:, 0] = np.repeat(rng.integers(1, n + 1, k // 32 + 1), 32)[:k]
    same = rand.copy()
    same[::3, 1] = same[::3, 0]  # u == v gives 0
    return {"random": rand, "one_u": one_u, "runs": runs, "same": same}


@pytest.mark.parametrize("n,m,deg", [(3, 4, 2), (300, 4000, 60), (2000, 160_000, 1900)])
def test_grouped_pairs_match_oracle(n, m, deg):
    A, B, _, init = bm.gen_pair(1 if n < 1000 else 3, n=n, m_target=m, max_degree=deg, seed=7)
    e = make_engine(n, (A.src, A.dst, A.w), (B.src, B.dst, B.w), init)
    orc = Oracle(n, (A.src, A.dst, A.w), (B.src, B.dst, B.w))
    for name, pairs in _lists(n, np.random.default_rng(n)).items():
        np.testing.assert_array_equal(e.delta_pairs(pairs), orc.pairs(init, pairs), err_msg=name)
    # a swap relabels the live lists that the grouped kernel streams
    u, v = 1, n
    e.apply_swaps(np.array([u, v], np.int32))
    pi = e.get_mapping()
    pairs = _lists(n, np.random.default_rng(n + 1))["random"]
    np.testing.assert_array_equal(e.delta_pairs(pairs), orc.pairs(pi, pairs))
    e.close()


@pytest.mark.parametrize("k", [1, 2, 9, 1184, 2369, 9471, 13001])
def test_short_lists_match_oracle(k):
    n = 2000
    A, B, _, init = bm.gen_pair(3, n=n, m_target=40_000, max_degree=1500, seed=3)
    e = make_engine(n, (A.src, A.dst, A.w), (B.src, B.dst, B.w), init)
    orc = Oracle(n, (A.src, A.dst, A.w), (B.src, B.dst, B.w))
    rng = np.random.default_rng(k)
    deg = np.bincount(A.src, minlength=n + 1) + np.bincount(A.dst, minlength=n + 1)
    hubs = np.argsort(-deg)[:20]
    pairs = rng.integers(1, n + 1, (k, 2)).astype(np.int32)
    pairs[::5, 0] = hubs[rng.integers(0, 20, len(pairs[::5]))]  # pairs that a whole block shares
    pairs[::7] = pairs[::7, ::-1]
    np.testing.assert_array_equal(e.delta_pairs(pairs), orc.pairs(init, pairs))
    e.close()


@pytest.mark.parametrize("mode", ["exact", "ref-cpu"])
def test_grouped_pairs_with_selfloops(golden_selfloop_ref, mode):
    g = golden_selfloop_ref
    n, A, B = golden_graphs(g)
    e = make_engine(n, A, B, g["pi_init"])
    e.set_semantics(mode)
    for name, pairs in _lists(n, np.random.default_rng(5)).items():
        np.testing.assert_array_equal(e.delta_pairs(pairs), _slices(e, pairs), err_msg=name)
    e.close()


def test_repeated_edges_stay_exact(golden_selfloop):
    g = golden_selfloop
    n, A, B = golden_graphs(g)
    pi = g["pis"][0]
    orc = Oracle(n, A, B)
    e = make_engine(n, A, B, pi)
    pairs = _lists(n, np.random.default_rng(6))["random"]
    exp = np.array([orc.exact_delta(pi, u, v) if u != v else 0 for u, v in pairs])
    np.testing.assert_array_equal(e.delta_pairs(pairs), exp)
    e.close()


@pytest.mark.parametrize("offset", [0, 4])
def test_device_pairs_bad_ids_and_alignment(offset):
    n = 300
    A, B, _, init = bm.gen_pair(1, n=n, m_target=4000, seed=9)
    e = make_engine(n, (A.src, A.dst, A.w), (B.src, B.dst, B.w), init)
    pairs = _lists(n, np.random.default_rng(8))["random"]
    exp = _slices(e, pairs)
    pairs[5] = (0, 7)
    pairs[6] = (7, n + 1)
    pairs[7] = (-3, 7)
    exp[5:8] = 0  # ids outside 1..n give 0
    d_p = e.dev_alloc(pairs.nbytes + 8)
    d_o = e.dev_alloc(8 * len(pairs))
    e.h2d(d_p + offset, pairs)
    e.delta_pairs_dev(d_p + offset, len(pairs), d_o)
    out = np.zeros(len(pairs), np.int64)
    e.d2h(out, d_o)
    e.sync()
    np.testing.assert_array_equal(out, exp)
    e.dev_free(d_p)
    e.dev_free(d_o)
    e.close()
