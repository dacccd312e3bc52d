"""Grouped pair deltas at the sizes where the kernel's shape changes: two blocks
an SM up to 12,479 vertices, one wide block above, and no tables that fit past
27,007; many more items than blocks, most of them claimed, against the oracle."""
import numpy as np
import pytest

import bmb200 as bm
from conftest import make_engine
from oracle_bind import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,grouped", [(12479, True), (12480, True), (27007, True), (27008, False)])
def test_shapes(n, grouped):
    A, B, _, init = bm.gen_pair(3, n=n, m_target=40 * n, max_degree=4000, seed=n)
    rng = np.random.default_rng(n)
    pairs = rng.integers(1, n + 1, (14 * n, 2)).astype(np.int32)
    pairs[:700, 0] = n  # several items of one u
    GA, GB = (A.src, A.dst, A.w), (B.src, B.dst, B.w)
    e = make_engine(n, GA, GB, init)
    before = e.launch_count()
    got = e.delta_pairs(pairs)
    assert (e.launch_count() - before > 1) == grouped
    np.testing.assert_array_equal(got, Oracle(n, GA, GB).pairs(init, pairs))
    for _ in range(3):  # the claims start anew with every call
        np.testing.assert_array_equal(e.delta_pairs(pairs), got)
    e.close()
