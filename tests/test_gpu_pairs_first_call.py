"""A context's first list of pairs grows its memory in one request at most, the
grouped kernel's sort included."""
import numpy as np
import pytest

import bmb200 as bm
from conftest import make_engine
from oracle_bind import Oracle

pytestmark = pytest.mark.gpu


# within the staging that loading the graphs left (41 bytes an edge), and past it
@pytest.mark.parametrize("k,calls", [(20_000, 0), (600_000, 2)])
def test_allocations_of_the_first_call(k, calls):
    n = 2000
    A, B, _, init = bm.gen_pair(3, n=n, m_target=160_000, max_degree=1900, seed=7)
    GA, GB = (A.src, A.dst, A.w), (B.src, B.dst, B.w)
    e = make_engine(n, GA, GB, init)
    pairs = np.random.default_rng(k).integers(1, n + 1, (k, 2)).astype(np.int32)
    allocs, launches = bm.cuda_lib().bm_alloc_count(), e.launch_count()
    got = e.delta_pairs(pairs)
    assert e.launch_count() - launches > 1  # grouped
    assert bm.cuda_lib().bm_alloc_count() - allocs == calls  # a release and an allocation
    np.testing.assert_array_equal(got[:20_000], Oracle(n, GA, GB).pairs(init, pairs[:20_000]))
    np.testing.assert_array_equal(e.delta_pairs(pairs), got)
    e.close()
