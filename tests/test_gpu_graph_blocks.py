"""Graphs that take over an earlier graph's block: results are those of a fresh
engine, also where captured row launches of the earlier graph are still there."""
import numpy as np
import pytest

import bmb200 as bm

pytestmark = pytest.mark.gpu

N = 600


def _graph(m, seed):
    """m distinct edges without self-loops."""
    r = np.random.default_rng(seed)
    e = r.choice(N * (N - 1), m, replace=False)
    src, dst = e // (N - 1) + 1, e % (N - 1) + 1
    dst += dst >= src
    return bm.Graph(N, src.astype(np.int32), dst.astype(np.int32), r.integers(1, 9, m).astype(np.int32))


@pytest.mark.parametrize("sizes", [(9000, 8300, 8900, 8200), (3000, 9000, 3100, 8800), (30_000, 9000, 29_000, 8500, 31_000)])
@pytest.mark.parametrize("side", [0, 1])
def test_replaced(sizes, side):
    fixed = _graph(9000, 1)
    pi = np.concatenate([[0], np.random.default_rng(2).permutation(N) + 1]).astype(np.int32)
    # more rows than a split launch takes, so that the launches are captured
    rows = (np.arange(300) % N + 1).astype(np.int32)
    with bm.Engine(0) as e:
        e.set_graph(1 - side, fixed)
        for k, m in enumerate(sizes):
            g = _graph(m, 10 + k)
            e.set_graph(side, g)
            e.set_mapping(pi)
            if k % 2 == 0 and k + 1 < len(sizes):
                continue  # replaced without a row launch of its own
            with bm.Engine(0) as fresh:
                fresh.set_graph(side, g)
                fresh.set_graph(1 - side, fixed)
                fresh.set_mapping(pi)
                assert e.score() == fresh.score()
                want = fresh.rows_best(rows)
                for _ in range(3):  # plain, captured, replayed
                    np.testing.assert_array_equal(e.rows_best(rows), want)
