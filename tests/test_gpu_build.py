"""The layout built on the device (edge lists of 8,192 entries and more)
against the host builder, which shorter lists take: the same graph with and
without zero-weight entries, which the layout drops, must behave the same.
Rejected inputs keep their errors and leave the graphs in place."""
import numpy as np
import pytest

import bmb200 as bm
from conftest import make_engine
from oracle_bind import Oracle

pytestmark = pytest.mark.gpu


def _edges(n, m, rng, dups, selfs):
    src, dst = rng.integers(1, n + 1, (2, m)).astype(np.int32)
    w = rng.integers(0, 30, m).astype(np.int32)  # some zero weights too
    hub = rng.random(m) < 0.2
    src[hub] = 1 + src[hub] % min(3, n)
    loops = src == dst
    dst[loops] = dst[loops] % n + 1
    if dups:
        k = m // 5
        src[-k:], dst[-k:] = src[:k], dst[:k]  # later entries of the same edges, other weights
    if selfs:
        v = rng.permutation(n)[:n // 4] + 1
        src = np.concatenate([v, src]).astype(np.int32)
        dst = np.concatenate([v, dst]).astype(np.int32)
        w = np.concatenate([rng.integers(1, 30, len(v)), w]).astype(np.int32)
    return src, dst, w


def _padded(n, G, rng, extra):
    """The same graph with zero-weight entries mixed in ahead of every entry
    of their edge (of equal edges in B the last counts)."""
    src, dst = rng.integers(1, n + 1, (2, extra)).astype(np.int32)
    loops = src == dst
    dst[loops] = dst[loops] % n + 1
    first = len(G[0]) // 2
    out = []
    for z, g in zip((src, dst, np.zeros(extra, np.int32)), G):
        out.append(np.concatenate([z[:extra // 2], g[:first], g[first:]]))
    # the rest ahead of the second half, on edges that do not occur
    key = set(zip(G[0].tolist(), G[1].tolist()))
    keep = np.array([(int(s), int(d)) not in key for s, d in zip(src[extra // 2:], dst[extra // 2:])])
    z = (src[extra // 2:][keep], dst[extra // 2:][keep], np.zeros(int(keep.sum()), np.int32))
    at = extra // 2 + first
    return tuple(np.concatenate([o[:at], q, o[at:]]).astype(np.int32) for o, q in zip(out, z))


@pytest.mark.parametrize("n,m", [(2, 5), (40, 700), (700, 6000), (3000, 7000)])
@pytest.mark.parametrize("dups,selfs", [(False, False), (True, False), (True, True)])
def test_device_build_equals_host_build(n, m, dups, selfs):
    rng = np.random.default_rng(n + m + 2 * dups + selfs)
    A, B = _edges(n, m, rng, dups, selfs), _edges(n, m, rng, dups, selfs)
    A2, B2 = _padded(n, A, rng, 20_000), _padded(n, B, rng, 20_000)
    assert len(A[0]) < 8192 <= len(A2[0]) and len(B2[0]) >= 8192
    pi = np.concatenate([[0], rng.permutation(n) + 1]).astype(np.int32)
    e, f = make_engine(n, A, B, pi), make_engine(n, A2, B2, pi)
    for side in (0, 1):
        assert e.graph_info(side) == f.graph_info(side)
    assert e.score() == f.score() == Oracle(n, A, B).score(pi)
    rows = np.arange(1, min(n, 200) + 1, dtype=np.int32)
    np.testing.assert_array_equal(e.delta_rows(rows), f.delta_rows(rows))
    pairs = rng.integers(1, n + 1, (500, 2)).astype(np.int32)
    np.testing.assert_array_equal(e.delta_pairs(pairs), f.delta_pairs(pairs))
    if n > 8:
        # draws and selections read the host copy of A's sorted lists
        for x, y in zip(e.perturb(4, mode=1, seed=3), f.perturb(4, mode=1, seed=3)):
            np.testing.assert_array_equal(x, y)
        pe, _ = e.search_batched(max_sweeps=2)
        pf, _ = f.search_batched(max_sweeps=2)
        assert pe.score == pf.score
        np.testing.assert_array_equal(e.get_mapping(), f.get_mapping())
    e.close()
    f.close()


@pytest.mark.parametrize("m", [8192, 12287, 12288, 12289, 40_000])
def test_tile_edges_match_oracle(m):
    n = 600
    rng = np.random.default_rng(m)
    key = rng.permutation(n * n)[:2 * m]
    s, d = (key // n + 1).astype(np.int32), (key % n + 1).astype(np.int32)
    s, d = s[s != d][:m], d[s != d][:m]
    A = (s, d, rng.integers(1, 99, m).astype(np.int32))
    B = (d, s, rng.integers(1, 32767, m).astype(np.int32))
    pi = np.concatenate([[0], rng.permutation(n) + 1]).astype(np.int32)
    e, orc = make_engine(n, A, B, pi), Oracle(n, A, B)
    assert e.score() == orc.score(pi)
    rows = np.array([1, 2, n // 2, n], np.int32)
    np.testing.assert_array_equal(e.delta_rows(rows), orc.rows(pi, rows))
    assert e.graph_info(0)["m"] == m
    e.close()


def test_rejected_inputs_leave_the_graphs():
    n, m = 20_000, 17_000
    rng = np.random.default_rng(1)
    A = (np.full(m, 1, np.int32), np.arange(2, m + 2, dtype=np.int32), np.full(m, 5, np.int32))
    e = make_engine(n, A, A, np.arange(n + 1))
    score = e.score()

    def bad(field, at, value):
        G = [x.copy() for x in A]
        G[field][at] = value
        return G

    heavy = [A[0], A[1], np.full(m, 32767, np.int32)]  # weighted degree 2^29 and more
    loops = [x.copy() for x in A]
    for k in (7, 9):
        loops[0][k] = loops[1][k] = 55
    for G, text in ((bad(0, 3, 0), "id outside"), (bad(1, m - 1, n + 1), "id outside"), (bad(2, 5, -1), "weight"),
                    (bad(2, 5, 32768), "weight"), (heavy, "weighted degree"), (loops, "more than one self-loop")):
        with pytest.raises(bm.BMError, match=text):
            e.set_graph(0, bm.Graph(n, *G))
    assert e.score() == score
    e.set_graph(1, bm.Graph(n, *heavy))  # only A is bounded
    e.set_mapping(np.arange(n + 1))
    assert e.score() == score
    e.close()
    del rng
