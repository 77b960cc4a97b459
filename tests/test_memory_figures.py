"""The library's memory figures against what it allocates (over the stand-in
runtime, tests/fake_cuda, which counts device allocations)."""
import ctypes as C

import numpy as np
import pytest

from tests import fake_cuda

BITARRAY, RANKSELECT, TREE = 0, 1, 2


@pytest.fixture(scope="module")
def L():
    return fake_cuda.load()


def needed(L, kind, n, arg, sigma=0):
    b = C.c_uint64()
    assert L.ewt_needed_memory(kind, n, arg, sigma, C.byref(b)) == 0
    return b.value


@pytest.mark.parametrize("bits,arrays", [(1, 1), (4097, 3), ((1 << 20) + 1, 200), (1 << 30, 1)])
@pytest.mark.parametrize("rate", [0, 32, 256])
def test_rank_select_bound(L, bits, arrays, rate):
    """EWT_MEM_RANKSELECT covers every sample rate, 32 being the densest (the
    handle's 16-byte status word aside)."""
    words = np.zeros((bits + 31) // 32 * arrays, np.uint32)
    sizes = np.full(arrays, bits, np.uint64)
    out = C.c_void_p()
    L.fake_reset()
    before = L.fake_live()
    assert L.ewt_rs_build(words.ctypes.data, sizes.ctypes.data_as(C.POINTER(C.c_uint64)), arrays, 0,
                          C.byref(out)) == 0
    assert L.ewt_rs_set_select_samples(out, rate) == 0
    held = L.fake_live() - before - 16
    assert L.ewt_rs_free(out) == 0
    assert held <= needed(L, RANKSELECT, bits, arrays)


def test_batch_shares(L):
    """The trees of a batch build that share a store count all of it between
    them (their small tables are padded to 256 bytes: seven per tree)."""
    rng = np.random.default_rng(3)
    texts = [np.zeros(n, np.uint8) for n in rng.integers(1 << 21, 1 << 22, 6)]
    al = np.arange(16, dtype=np.uint8)
    ptr = lambda arrays: (C.c_void_p * len(arrays))(*[a.ctypes.data for a in arrays])
    lens = np.array([t.size for t in texts], np.uint64)
    sigmas = np.full(len(texts), 16, np.uint64)
    out = (C.c_void_p * len(texts))()
    L.fake_reset()
    before = L.fake_live()
    assert L.ewt_build_batch(ptr(texts), lens.ctypes.data, len(texts), 1, ptr([al] * len(texts)),
                             sigmas.ctypes.data, 0, out, None) == 0
    held = L.fake_live() - before
    from ecl_wavelet_gb300 import Info
    total = 0
    for t in out:
        i = Info()
        assert L.ewt_get_info(t, C.byref(i)) == 0
        total += i.device_bytes
    for t in out:
        assert L.ewt_free(t) == 0
    assert held - 7 * 256 * len(texts) <= total <= held + held // 100
