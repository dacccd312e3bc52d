"""The delta table built from one-sided gains (forced, whatever the size) against
the row kernel's own finish and against whole rows, around its 64 x 64 tiles,
with wider rows and other starts, self-loops and repeated edges on both sides."""
import numpy as np
import pytest

from conftest import golden_graphs, make_engine

pytestmark = pytest.mark.gpu


def _table(e, n, ld, shift):
    """The table at an offset of `shift` ints, what is not its own filled; the launches."""
    size = (n + 1) * ld
    host = np.full(size + shift, 77, np.int32)
    d = e.dev_alloc(host.nbytes)
    e.h2d(d, host)
    before = e.launch_count()
    e.delta_table_dev(d + 4 * shift, ld)
    launches = e.launch_count() - before
    e.sync()
    e.d2h(host, d)
    e.sync()
    e.dev_free(d)
    assert (host[:shift] == 77).all()
    return host[shift:].reshape(n + 1, ld), launches


def _check(e, n, ld, shift=0, one_sided=True):
    rows = e.delta_rows(np.arange(1, n + 1, dtype=np.int32))
    launches = []
    for mode in (1, -1):
        e.set_path("table_gains", mode)
        tab, count = _table(e, n, ld, shift)
        np.testing.assert_array_equal(tab[1:, :n + 1], rows)
        assert not tab[0].any()
        assert (tab[1:, n + 1:] == 77).all()  # columns past n are not the table's
        launches.append(count)
    assert (launches[0] > launches[1]) == one_sided


def _edges(n, rng, repeats):
    m = 6 * n
    src, dst = rng.integers(1, n + 1, (2, m)).astype(np.int32)
    keep = src != dst
    loops = rng.permutation(n)[:n // 3].astype(np.int32) + 1
    src, dst = np.concatenate([src[keep], loops]), np.concatenate([dst[keep], loops])
    if repeats:
        k = int(keep.sum())
        src, dst = np.concatenate([src, src[:k // 2]]), np.concatenate([dst, dst[:k // 2]])
    return src, dst, rng.integers(1, 40, len(src)).astype(np.int32)


@pytest.mark.parametrize("repeats", [False, True])
@pytest.mark.parametrize("n", [2, 3, 4, 31, 62, 63, 64, 65, 126, 127, 128, 129, 191, 300, 577])
def test_tile_edges(n, repeats):
    rng = np.random.default_rng(2 * n + repeats)
    e = make_engine(n, _edges(n, rng, repeats), _edges(n, rng, True), np.concatenate([[0], rng.permutation(n) + 1]))
    ld = (n + 1 + 3) & ~3
    _check(e, n, ld)
    _check(e, n, ld + 4)
    _check(e, n, ld + 64, shift=4)
    _check(e, n, ld + 1, one_sided=False)  # rows not 16-byte aligned
    _check(e, n, ld, shift=1, one_sided=False)
    u, v = rng.integers(1, n + 1, 2)
    e.apply_swaps(np.array([u, v], np.int32))
    _check(e, n, ld)
    e.set_semantics("ref-cpu")
    _check(e, n, ld, one_sided=n // 3 == 0)  # its self-loop terms are per row
    e.close()


def test_golden_graphs(golden_selfloop, golden_selfloop_ref):
    for g, pi in ((golden_selfloop_ref, golden_selfloop_ref["pi_init"]), (golden_selfloop, golden_selfloop["pis"][0])):
        n, A, B = golden_graphs(g)
        e = make_engine(n, A, B, pi)
        _check(e, n, (n + 1 + 3) & ~3)
        e.close()


def test_no_edges():
    none = tuple(np.zeros(0, np.int32) for _ in range(3))
    n = 70
    e = make_engine(n, none, none, np.arange(n + 1, dtype=np.int32))
    _check(e, n, 72)
    e.close()
