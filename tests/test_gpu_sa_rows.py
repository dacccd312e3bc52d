"""Annealing chains whose B rows fall on every side of the index's limits
(shared slots, more than 252 entries, more than the staging buffer), and a
mapping too large for shared memory, replayed on the CPU."""
import numpy as np
import pytest

import bmb200 as bm
from oracle_bind import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m,deg", [(2, 2, 1), (600, 90_000, 400), (3000, 120_000, 2500), (9000, 200_000, 3000),
                                     (40_000, 120_000, 600)])
@pytest.mark.parametrize("threads", [256, 512])
def test_rows_of_every_length_replay(n, m, deg, threads):
    A, B, _, init = bm.gen_pair(1 if n == 2 else 3, n=n, m_target=m, max_degree=deg, seed=n)
    eng = bm.Engine(0)
    batch = bm.Batch(eng)
    batch.add_pair(A, B)
    steps = 3000
    pis, scores, acc, _ = batch.sa_run([0, 0], [5, 6], [init, init], steps, t0=50.0, t_end=0.01, candidates=8,
                                       threads=threads)
    orc = Oracle(n, (A.src, A.dst, A.w), (B.src, B.dst, B.w))
    for c, key in enumerate((5, 6)):
        pi_o, s_o, a_o = orc.sa(init, key, steps, 50.0, 0.01)
        np.testing.assert_array_equal(pis[c], pi_o)
        assert scores[c] == s_o and acc[c] == a_o
    batch.close()
    eng.close()
