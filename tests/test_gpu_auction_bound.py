"""The auction's clock bound running out anywhere in a solve, in the rounds with
one bidder above all (most rounds of a sparse matrix): the call returns
BM_TIMEOUT, and the next one on the same context solves the matrix."""
import numpy as np
import pytest

import bmb200 as bm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [200, 300, 1025])  # one block; a cluster of blocks
def test_bound_runs_out_between_rounds(k):
    rng = np.random.default_rng(k)
    a = np.where(rng.random((k, k)) < 0.02, rng.integers(1, 2000, (k, k)), 0).astype(np.int32)
    with bm.Engine(0) as e:
        total = e.lap_solve(a)[1]
        ended = []
        for limit in np.geomspace(5e3, 5e7, 60).astype(np.int64):
            assert e.L.bm_set_wait_limit(e.h, int(limit)) == bm.BM_OK
            try:
                ended.append(e.lap_solve(a)[1])
            except bm.BMError as ex:
                assert ex.status == bm.BM_TIMEOUT
                ended.append(None)
        assert e.L.bm_set_wait_limit(e.h, 0) == bm.BM_OK
        assert ended[0] is None and all(t in (None, total) for t in ended)
        late = [t for t in ended if t is None]
        assert len(late) >= 3  # some of them ran out well inside the solve
        assign, again = e.lap_solve(a)
        assert again == total
        assert sorted(assign.tolist()) == list(range(k))
