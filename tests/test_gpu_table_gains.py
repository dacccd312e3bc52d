"""The delta table built from one-sided gains, at sizes around its 64 x 64
tiles, against whole rows (which the row tests hold against the oracle), with
self-loops and repeated edges, and with layouts that take the row kernel's own
finish."""
import numpy as np
import pytest

import bmb200 as bm
from conftest import golden_graphs, make_engine

pytestmark = pytest.mark.gpu


def _table(e, n, ld, shift=0):
    """The table as built at an offset of `shift` ints, padding columns filled."""
    size = (n + 1) * ld
    host = np.full(size + shift, 77, np.int32)
    d = e.dev_alloc(4 * (size + shift))
    e.h2d(d, host)
    e.delta_table_dev(d + 4 * shift, ld)
    e.sync()
    e.d2h(host, d)
    e.sync()
    e.dev_free(d)
    return host[shift:].reshape(n + 1, ld)


def _check(e, n, ld, shift=0):
    tab = _table(e, n, ld, shift)
    rows = np.arange(1, n + 1, dtype=np.int32)
    np.testing.assert_array_equal(tab[1:, :n + 1], e.delta_rows(rows))
    assert not tab[0].any()
    assert (tab[1:, n + 1:] == 77).all()  # columns past n are not the table's


@pytest.mark.parametrize("n", [2, 3, 4, 31, 62, 63, 64, 65, 127, 128, 129, 300, 577])
def test_tile_edges(n):
    rng = np.random.default_rng(n)
    m = 6 * n
    src, dst = rng.integers(1, n + 1, (2, m)).astype(np.int32)
    keep = src != dst
    w = rng.integers(1, 40, m).astype(np.int32)
    A = (src[keep], dst[keep], w[keep])
    B = (dst[keep], src[keep], w[keep][::-1].copy())
    e = make_engine(n, A, B, np.concatenate([[0], rng.permutation(n) + 1]))
    ld = (n + 1 + 3) & ~3
    _check(e, n, ld)
    _check(e, n, ld + 8)
    _check(e, n, ld + 1)  # rows not 16-byte aligned: the row kernel's finish
    _check(e, n, ld, shift=1)
    u, v = rng.integers(1, n + 1, 2)
    e.apply_swaps(np.array([u, v], np.int32))
    _check(e, n, ld)
    e.close()


@pytest.mark.parametrize("mode", ["exact", "ref-cpu"])
def test_selfloops_and_repeats(golden_selfloop, golden_selfloop_ref, mode):
    for g, pi in ((golden_selfloop_ref, golden_selfloop_ref["pi_init"]), (golden_selfloop, golden_selfloop["pis"][0])):
        n, A, B = golden_graphs(g)
        e = make_engine(n, A, B, pi)
        e.set_semantics(mode)
        _check(e, n, (n + 1 + 3) & ~3)
        e.close()
