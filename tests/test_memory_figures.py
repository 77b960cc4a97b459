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
