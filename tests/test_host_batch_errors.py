"""A host batch that fails half-way has nothing of its own left on the GPU when
it returns: its kernels read and write the caller's buffers.  Over the
stand-in runtime (tests/fake_cuda): every call that the batch makes fails once,
for pageable buffers copied by kernels, used in place, and pinned ones."""
import ctypes as C

import numpy as np
import pytest

from tests import fake_cuda

UNREGISTERED, HOST = 0, 1  # cudaMemoryType


@pytest.fixture(scope="module")
def L():
    return fake_cuda.load()


def batches(L, tree, rs, m):
    q = np.zeros((m, 2), np.uint64)
    out = np.zeros(m, np.uint64)
    types = np.zeros(m, np.uint8)
    yield "rank", lambda: L.ewt_rank(tree, q.ctypes.data, m, out.ctypes.data)
    yield "mixed", lambda: L.ewt_mixed(tree, types.ctypes.data, q.ctypes.data, m, out.ctypes.data)
    if m <= 262_144:
        yield "noalloc", lambda: L.ewt_mixed_noalloc(tree, types.ctypes.data, q.ctypes.data, m,
                                                     out.ctypes.data)
    one, of = (C.c_void_p * 1)(tree.value), np.zeros(m, np.uint32)
    yield "multi", lambda: L.ewt_mixed_multi(one, 1, of.ctypes.data, types.ctypes.data,
                                             q.ctypes.data, m, out.ctypes.data)
    yield "rs", lambda: L.ewt_rs_rank(rs, 0, 1, q.ctypes.data, m, out.ctypes.data)


@pytest.mark.parametrize("host_type,m", [(UNREGISTERED, 1 << 19), (UNREGISTERED, 100),
                                                  (HOST, 1 << 21)])
@pytest.mark.parametrize("call", ["launch", "cudaEventRecord", "cudaStreamWaitEvent",
                                  "cudaMemcpyAsync", "cudaMemsetAsync", "occupancy"])
def test_nothing_left_behind(L, call, host_type, m):
    L.fake_reset()
    L.fake_set(b"host_type", UNREGISTERED)
    tree = fake_cuda.build(L, np.zeros(1000, np.uint8), np.arange(2, dtype=np.uint8))
    rs = C.c_void_p()
    words, bits = np.zeros(32, np.uint32), np.array([1000], np.uint64)
    assert L.ewt_rs_build(words.ctypes.data, bits.ctypes.data_as(C.POINTER(C.c_uint64)), 1, 0,
                          C.byref(rs)) == 0
    L.fake_set(b"host_type", host_type)
    for name, run in batches(L, tree, rs, m):
        assert run() == 0, name
        assert L.fake_pending() == 0
        for n in range(1, 200):
            L.fake_fail(call.encode(), n)
            if run() == 0:  # all of its calls have failed once
                break
            assert L.fake_pending() == 0, (name, call, n)
        else:
            pytest.fail("the batch makes more calls than that")
        L.fake_fail(call.encode(), 0)
        assert run() == 0, name
    L.fake_set(b"host_type", UNREGISTERED)
    assert L.ewt_free(tree) == 0 and L.ewt_rs_free(rs) == 0
