"""The greedy matching's bit rows and shortlists at their edges: hubs beside
light vertices around the 128 bits of a row word and more words than threads,
duplicate edges and self-loops, and more vertices of one shape than a shortlist
has entries, against the host restatement."""
import numpy as np
import pytest

import bmb200 as bm

pytestmark = pytest.mark.gpu


def _hubs(n, seed, hubs, spokes):
    """`hubs` vertices with about `spokes` neighbours each way, the rest sparse."""
    r = np.random.default_rng(seed)
    h = r.permutation(n)[:hubs] + 1
    far = r.integers(1, n + 1, (2, hubs, spokes))
    src = np.concatenate([np.repeat(h, spokes), far[0].ravel(), r.integers(1, n + 1, 3 * n), h, h])
    dst = np.concatenate([far[1].ravel(), np.repeat(h, spokes), r.integers(1, n + 1, 3 * n), h, h])
    return bm.Graph(n, src.astype(np.int32), dst.astype(np.int32), np.ones(len(src), np.int32))


@pytest.mark.parametrize("n,hubs,spokes", [(127, 5, 64), (128, 6, 80), (129, 128, 70), (1024, 1, 65), (2049, 40, 900),
                                           (6400, 60, 101), (33000, 12, 3000)])
def test_rows(n, hubs, spokes):
    A, B = _hubs(n, n, hubs, spokes), _hubs(n, n + 1, hubs, spokes)
    with bm.Engine(0) as e:
        np.testing.assert_array_equal(e.greedy_match(A, B), bm.greedy_match(A, B))


@pytest.mark.parametrize("n", [63, 64, 65, 130, 2048])
def test_one_shape(n):
    """Every shortlist is the same, and most are used up."""
    ids = np.arange(1, n + 1, dtype=np.int32)
    ring = bm.Graph(n, ids, np.roll(ids, 1), np.ones(n, np.int32))
    with bm.Engine(0) as e:
        np.testing.assert_array_equal(e.greedy_match(ring, _hubs(n, n, 1, 20)), bm.greedy_match(ring, _hubs(n, n, 1, 20)))
        np.testing.assert_array_equal(e.greedy_match(ring, ring), ids_pi(n))


def ids_pi(n):
    return np.arange(n + 1, dtype=np.int32)
