"""When the batched search takes the gain tables, on the full-scale pair: for a
search over all rows that has come to accept few swaps, not for one over a few
rows, whose passes cost less than filling the tables; the same results with and
without them."""
import numpy as np
import pytest

import bmb200 as bm
from conftest import make_engine

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pair():
    A, B, _, init = bm.gen_pair(2)
    return A.n, (A.src, A.dst, A.w), (B.src, B.dst, B.w), init


def _search(pair, mode, rows, passes):
    e = make_engine(*pair)
    e.set_path("gain_tables", mode)
    before = e.launch_count()
    p, _ = e.search_batched(rows, max_sweeps=passes)
    got = p.accepts, p.score, p.rows_done, p.sweeps, p.converged, e.get_mapping().tobytes()
    launches = e.launch_count() - before
    e.close()
    return got, launches


def test_all_rows(pair):
    with_rule, used = _search(pair, 0, None, -1)
    without, plain = _search(pair, -1, None, -1)
    assert with_rule == without
    assert used != plain


@pytest.mark.parametrize("count", [1, 64, 600])
def test_a_few_rows(pair, count):
    rows = (np.random.default_rng(count).permutation(pair[0])[:count] + 1).astype(np.int32)
    with_rule, used = _search(pair, 0, rows, 6)
    without, plain = _search(pair, -1, rows, 6)
    assert with_rule == without
    assert with_rule[3] > 1  # a second pass was made, with or without them
    assert used == plain
