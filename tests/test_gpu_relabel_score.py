"""Relabelled bank-spread lists and the score at list lengths around a whole
turn of 128 positions, with balanced and unbalanced banks and a hub, against
the oracle (whole rows read every relabelled list, swaps its twins)."""
import numpy as np
import pytest

import bmb200 as bm
from conftest import make_engine
from oracle_bind import Oracle

pytestmark = pytest.mark.gpu


def _graph(n, rng, lengths, step):
    """Vertex v gets lengths[v] out-edges; step 32 keeps the ids of a list in
    few banks, step 1 spreads them over all."""
    src, dst = [], []
    for v, k in enumerate(lengths, start=1):
        ids = (rng.permutation(n // step)[:k] * step + int(rng.integers(step))) % n + 1
        ids = np.unique(ids[ids != v])
        src.append(np.full(len(ids), v))
        dst.append(ids)
    src, dst = np.concatenate(src).astype(np.int32), np.concatenate(dst).astype(np.int32)
    return src, dst, rng.integers(1, 50, len(src)).astype(np.int32)


@pytest.mark.parametrize("step", [1, 8, 32])
def test_lists_around_whole_turns(step):
    n = 9000 if step == 32 else 2000
    rng = np.random.default_rng(step)
    lengths = np.zeros(n, np.int64)
    sizes = [1, 2, 3, 4, 5, 31, 32, 33, 127, 128, 129, 130, 255, 256, 257, 700, 1999 // step]
    lengths[rng.permutation(n)[:len(sizes) * 8]] = np.repeat(sizes, 8)
    A, B = _graph(n, rng, lengths, step), _graph(n, rng, rng.permutation(lengths), step)
    pi = np.concatenate([[0], rng.permutation(n) + 1]).astype(np.int32)
    e = make_engine(n, A, B, pi)
    orc = Oracle(n, A, B)
    assert e.score() == orc.score(pi)
    rows = rng.permutation(n)[:24] + 1
    rows[:8] = np.argsort(-lengths)[:8] + 1
    rows = rows.astype(np.int32)
    np.testing.assert_array_equal(e.delta_rows(rows), orc.rows(pi, rows))
    for u, v in rng.integers(1, n + 1, (6, 2)):
        if u != v:
            e.apply_swaps(np.array([u, v], np.int32))
    pi = e.get_mapping()
    assert e.score() == orc.score(pi)
    np.testing.assert_array_equal(e.delta_rows(rows), orc.rows(pi, rows))
    # the overlap at both ends of every entry: twice the score without self-loops
    assert int(e.overlap().astype(np.int64).sum()) == 2 * e.score()
    e.close()


def test_score_of_one_hub_and_empty_lists():
    n = 5000  # one list of many stretches, all others empty
    rng = np.random.default_rng(4)
    dst = np.arange(2, n + 1, dtype=np.int32)
    A = (np.ones(n - 1, np.int32), dst, rng.integers(1, 9, n - 1).astype(np.int32))
    B = (np.ones(n - 1, np.int32), dst, rng.integers(1, 9, n - 1).astype(np.int32))
    pi = np.concatenate([[0, 1], rng.permutation(n - 1) + 2]).astype(np.int32)
    e = make_engine(n, A, B, pi)
    assert e.score() == Oracle(n, A, B).score(pi)
    e.close()
