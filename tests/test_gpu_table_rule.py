"""The delta table on both sides of the rule that keeps small ones on the row
kernel's own finish, with self-loops and repeated edges, against whole rows; the
one-sided build around its 64 x 64 tiles."""
import numpy as np
import pytest

from conftest import make_engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(700, 1000), (700, 180_000), (1999, 4000), (2000, 4000), (2047, 6000), (2048, 6000),
                                 (2049, 9000), (2113, 200_000), (2999, 4000), (3000, 4000), (3007, 5000), (3008, 5000),
                                 (3009, 5000)])
def test_both_sides(n, m):
    rng = np.random.default_rng(n + m)

    def edges(repeats):
        src, dst = rng.integers(1, n + 1, (2, m)).astype(np.int32)
        keep = src != dst
        loops = rng.permutation(n)[:n // 4].astype(np.int32) + 1  # one self-loop a vertex at most
        src, dst = np.concatenate([src[keep], loops]), np.concatenate([dst[keep], loops])
        if repeats:
            src, dst = np.concatenate([src, src[:50]]), np.concatenate([dst, dst[:50]])
        return src, dst, rng.integers(1, 40, len(src)).astype(np.int32)

    e = make_engine(n, edges(False), edges(True), np.concatenate([[0], rng.permutation(n) + 1]))
    ld = (n + 1 + 3) & ~3
    host = np.full((n + 1, ld), 77, np.int32)
    d = e.dev_alloc(host.nbytes)
    for _ in range(2):
        e.h2d(d, host)
        e.delta_table_dev(d, ld)
        e.sync()
        tab = np.empty_like(host)
        e.d2h(tab, d)
        e.sync()
        np.testing.assert_array_equal(tab[1:, :n + 1], e.delta_rows(np.arange(1, n + 1, dtype=np.int32)))
        assert not tab[0].any()
        assert (tab[1:, n + 1:] == 77).all()
        e.apply_swaps(rng.permutation(n)[:2].astype(np.int32) + 1)
    e.dev_free(d)
    e.close()
