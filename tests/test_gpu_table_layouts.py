"""The best pairs of a delta table in any layout that bm_delta_table_dev fills:
every stride from n + 1 on and any start, 16-byte boundaries or not."""
import numpy as np
import pytest

import bmb200 as bm
from conftest import make_engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 5, 64, 300, 2111])
def test_topk(n):
    A, B, _, init = bm.gen_pair(1, n=n, m_target=min(12 * n, n * (n - 1) // 2), max_degree=max(2, n // 4), seed=n)
    e = make_engine(n, (A.src, A.dst, A.w), (B.src, B.dst, B.w), init)
    rows = e.delta_rows(np.arange(1, n + 1, dtype=np.int32))
    u, v = np.triu_indices(n + 1, 1)
    u, v = u[u > 0], v[u > 0]
    order = np.lexsort((v, u, -rows[u - 1, v]))
    d = e.dev_alloc(4 * ((n + 1) * (n + 9) + 8))
    for extra in range(8):
        ld = n + 1 + extra
        for shift in (0, 1, 2, 3):
            tab = d + 4 * shift
            e.delta_table_dev(tab, ld)
            for k in (1, 7, min(len(u), 900)):
                k = min(k, len(u))
                pairs, deltas = e.table_topk(tab, ld, k)
                best = order[:k]
                np.testing.assert_array_equal(pairs, np.stack([u[best], v[best]], 1))
                np.testing.assert_array_equal(deltas, rows[u[best] - 1, v[best]])
    e.dev_free(d)
    e.close()


def test_search_on_an_unaligned_table():
    n = 301
    A, B, _, init = bm.gen_pair(1, n=n, m_target=4000, max_degree=80, seed=3)
    GA, GB = (A.src, A.dst, A.w), (B.src, B.dst, B.w)
    got = []
    for ld, shift in ((304, 0), (302, 3)):
        e = make_engine(n, GA, GB, init)
        d = e.dev_alloc(4 * ((n + 1) * ld + 8))
        e.delta_table_dev(d + 4 * shift, ld)
        p, _ = e.search_table(d + 4 * shift, ld, k=64)
        got.append((p.score, p.accepts, e.get_mapping().tolist()))
        e.dev_free(d)
        e.close()
    assert got[0] == got[1]
