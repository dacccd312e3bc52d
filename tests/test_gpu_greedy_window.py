"""The windowed greedy matching at its edges: vertex counts around the 32
vertices held at once and the 1,024 commits between compactions, features that
all tie, and sums far apart, against the host restatement."""
import numpy as np
import pytest

import bmb200 as bm

pytestmark = pytest.mark.gpu


def _equal(A, B):
    with bm.Engine(0) as e:
        np.testing.assert_array_equal(e.greedy_match(A, B), bm.greedy_match(A, B))


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 1023, 1025, 2100, 3300])
@pytest.mark.parametrize("kind", ["ring", "random", "stars", "lopsided"])
def test_edges(n, kind):
    rng = np.random.default_rng(n)
    ids = np.arange(1, n + 1, dtype=np.int32)

    def graph(seed, shape):
        r = np.random.default_rng(seed)
        if shape == "ring":  # every vertex has the same features
            src, dst = ids, np.roll(ids, 1)
        elif shape == "stars":  # few distinct features, far apart
            src, dst = np.minimum(ids, 1 + ids % 3), r.permutation(ids)
        else:
            m = 4 * n
            src, dst = r.integers(1, n + 1, (2, m))
        src, dst = np.asarray(src, np.int32), np.asarray(dst, np.int32)
        return bm.Graph(n, src, dst, np.ones(len(src), np.int32))

    A = graph(n + 1, "ring" if kind == "lopsided" else kind)
    _equal(A, graph(n + 2, "random" if kind == "lopsided" else kind))
    del rng
