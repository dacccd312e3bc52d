"""bm_delta_pairs_dev on the context's stream as its callers may use it: captured
into a graph of their own that is replayed after larger calls, and enqueued
behind work that is still running, also when its scratch has to grow."""
import ctypes as C

import numpy as np
import pytest

import bmb200 as bm
from conftest import make_engine

pytestmark = pytest.mark.gpu

NOT_READY = 600
N = 2000


@pytest.fixture(scope="module")
def drv():
    return C.CDLL("libcuda.so.1")


def _chk(status):
    assert status == 0, status


class _Pairs:
    """Device buffers of one list of pairs."""

    def __init__(self, e, k, seed):
        self.e, self.k = e, k
        self.host = np.random.default_rng(seed).integers(1, N + 1, (k, 2)).astype(np.int32)
        self.d_p, self.d_o = e.dev_alloc(8 * k), e.dev_alloc(8 * k)
        e.h2d(self.d_p, self.host)
        e.sync()

    def launch(self):
        self.e.delta_pairs_dev(self.d_p, self.k, self.d_o)

    def read(self):
        out = np.zeros(self.k, np.int64)
        self.e.d2h(out, self.d_o)
        self.e.sync()
        return out

    def free(self):
        self.e.dev_free(self.d_p)
        self.e.dev_free(self.d_o)


@pytest.fixture
def eng():
    A, B, _, init = bm.gen_pair(3, n=N, m_target=160_000, max_degree=1900, seed=7)
    e = make_engine(N, (A.src, A.dst, A.w), (B.src, B.dst, B.w), init)
    yield e
    e.close()


def test_captured_call_uses_no_scratch(eng, drv):
    stream = C.c_void_p(eng.L.bm_ctx_stream(eng.h))
    p, big = _Pairs(eng, 20_000, 1), _Pairs(eng, 400_000, 2)
    p.launch()  # the scratch of this size is in place
    good = p.read()
    before = eng.launch_count()
    _chk(drv.cuStreamBeginCapture_v2(stream, 1))  # thread-local mode
    p.launch()
    graph, ex = C.c_void_p(), C.c_void_p()
    _chk(drv.cuStreamEndCapture(stream, C.byref(graph)))
    assert eng.launch_count() == before + 1  # the kernel that needs none
    _chk(drv.cuGraphInstantiateWithFlags(C.byref(ex), graph, C.c_ulonglong(0)))
    big.launch()  # grows the scratch
    want = big.read()
    eng.h2d(p.d_o, np.zeros(p.k, np.int64))
    eng.sync()
    _chk(drv.cuGraphLaunch(ex, stream))
    big.launch()
    np.testing.assert_array_equal(p.read(), good)
    np.testing.assert_array_equal(big.read(), want)
    _chk(drv.cuGraphExecDestroy(ex))
    _chk(drv.cuGraphDestroy(graph))
    p.free()
    big.free()


def test_growing_call_does_not_wait(eng, drv):
    lists = [_Pairs(eng, k, k) for k in (16_000, 40_000, 120_000, 500_000)]
    lists[0].launch()  # the kernels are loaded
    lists[0].read()
    ld = (N + 1 + 3) & ~3
    tab = eng.dev_alloc(4 * (N + 1) * ld)
    eng.delta_table_dev(tab, ld)
    eng.sync()
    ev = eng.event()
    pending = []
    for p in lists[1:]:
        for _ in range(80):  # some ten milliseconds
            eng.delta_table_dev(tab, ld)
        eng.record(ev)
        p.launch()
        pending.append(drv.cuEventQuery(C.c_void_p(ev)) == NOT_READY)
    eng.sync()
    assert all(pending), pending
    for p in lists:
        grouped = p.read()
        part = np.concatenate([eng.delta_pairs(p.host[i:i + 1000]) for i in range(0, 16_000, 1000)])
        np.testing.assert_array_equal(grouped[:16_000], part)
        p.free()
    eng.dev_free(tab)
