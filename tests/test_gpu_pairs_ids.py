"""bm_delta_pairs refuses ids outside 1..n wherever in the list one is, names the
first, and leaves the caller's deltas as they are."""
import numpy as np
import pytest

import bmb200 as bm
from conftest import make_engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [0, -1, 301, 302, 600, 2**31 - 1, -2**31, -2**31 + 1, -301])
@pytest.mark.parametrize("k,at", [(1, 0), (1, 1), (3, 4), (500, 0), (500, 517), (500, 999)])
def test_bad_id(value, k, at):
    n = 300
    A, B, _, init = bm.gen_pair(1, n=n, m_target=3000, seed=2)
    e = make_engine(n, (A.src, A.dst, A.w), (B.src, B.dst, B.w), init)
    pairs = np.tile(np.array([1, n], np.int32), (k, 1))
    good = e.delta_pairs(pairs)
    assert (good == good[0]).all()
    pairs.reshape(-1)[at] = value
    out = np.full(k, 77, np.int64)
    st = e.L.bm_delta_pairs(e.h, pairs.ctypes.data, k, out.ctypes.data)
    assert st == bm.BM_INVALID_ARG
    assert f"pair entry {at} = {value} outside 1..{n}".encode() in e.L.bm_ctx_last_error(e.h)
    assert (out == 77).all()
    e.close()
