"""Grouped pair deltas (forced, whatever the list) against the ungrouped kernel
and the oracle: lists around an item's 256 pairs, both shapes of the kernel,
self-loops under both delta semantics, repeated edges, many lists in a row."""
import numpy as np
import pytest

import bmb200 as bm
from conftest import golden_graphs, make_engine
from oracle_bind import Oracle

pytestmark = pytest.mark.gpu


def _both(e, pairs, grouped=True):
    got = []
    for mode in (1, -1):
        e.set_path("pair_groups", mode)
        before = e.launch_count()
        got.append(e.delta_pairs(pairs))
        assert (e.launch_count() - before > 1) == (grouped and mode > 0)
    np.testing.assert_array_equal(got[0], got[1])
    return got[0]


@pytest.mark.parametrize("n", [2, 7, 8, 500, 12479, 12480])
def test_list_lengths(n):
    A, B, _, init = bm.gen_pair(3, n=n, m_target=min(30 * n, n * (n - 1) // 2), max_degree=max(2, n // 3), seed=n)
    GA, GB = (A.src, A.dst, A.w), (B.src, B.dst, B.w)
    e, orc, rng = make_engine(n, GA, GB, init), Oracle(n, GA, GB), np.random.default_rng(n)
    hub = 1 + int(np.argmax(np.bincount(A.src, minlength=n + 1)[1:]))
    for k in (1, 2, 31, 33, 255, 256, 257, 513, 2600, 5000):
        pairs = rng.integers(1, n + 1, (k, 2)).astype(np.int32)
        pairs[k // 3:, 0] = hub  # one u with several items, its lists cut into units
        pairs[::5] = pairs[::5, ::-1]
        np.testing.assert_array_equal(_both(e, pairs), orc.pairs(init, pairs), err_msg=str(k))
    u, v = 1, n
    e.apply_swaps(np.array([u, v], np.int32))
    pairs = rng.integers(1, n + 1, (1000, 2)).astype(np.int32)
    np.testing.assert_array_equal(_both(e, pairs), orc.pairs(e.get_mapping(), pairs))
    e.close()


@pytest.mark.parametrize("semantics", ["exact", "ref-cpu"])
def test_selfloops(golden_selfloop_ref, semantics):
    g = golden_selfloop_ref
    n, A, B = golden_graphs(g)
    e = make_engine(n, A, B, g["pi_init"])
    e.set_semantics(semantics)
    _both(e, np.random.default_rng(5).integers(1, n + 1, (700, 2)).astype(np.int32))
    e.close()


def test_repeated_edges_are_not_grouped(golden_selfloop):
    g = golden_selfloop
    n, A, B = golden_graphs(g)
    e = make_engine(n, A, B, g["pis"][0])
    _both(e, np.random.default_rng(6).integers(1, n + 1, (3000, 2)).astype(np.int32), grouped=False)
    e.close()
