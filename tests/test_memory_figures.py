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


def zeros(nbytes, shift=0):
    """Reserved, untouched address space, `shift` bytes past a page."""
    import mmap
    m = mmap.mmap(-1, nbytes + shift, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS | 0x4000)
    return np.frombuffer(m, np.uint8)[shift:]


def build_peak(L, dtype, sigma, n, copied, short):
    """Device bytes at the peak of a build; copied: the text starts off a
    16-byte boundary, so that the device gets a copy; short: but for 1,000 symbols of
    the longest code the text holds the first of the short ones."""
    size = np.dtype(dtype).itemsize
    text = zeros(n * size, size if copied else 0)
    al = np.arange(sigma, dtype=np.uint64).astype(dtype)
    bits = max(1, (sigma - 1).bit_length())
    L.fake_reset()
    for entries in {(1 << bits) + 1, sigma + 1}:
        if short:
            L.fake_patch(entries * 8, 1, 1000)
        L.fake_patch(entries * 8, (1 << bits) // 2 + 1 if short else entries - 1, n)
    out = C.c_void_p()
    before = L.fake_live()
    assert L.ewt_build(text.ctypes.data, n, size, al.ctypes.data, sigma, 0, C.byref(out)) == 0, \
        L.ewt_last_error()
    peak = L.fake_peak() - before
    assert L.ewt_free(out) == 0
    return peak


GPU_BYTES = 284_208 << 20


@pytest.mark.parametrize("dtype,sigma,n,copied,short", [
    (np.uint8, 96, 73_000_000_000, 1, 0), (np.uint8, 96, 73_000_000_000, 1, 1),
    (np.uint8, 129, 72_000_000_000, 1, 0), (np.uint8, 129, 72_000_000_000, 0, 1),
    (np.uint8, 256, 57_000_000_000, 1, 0), (np.uint16, 1000, 40_000_000_000, 1, 0),
    (np.uint16, 33_024, 36_000_000_000, 1, 0), (np.uint16, 33_024, 36_000_000_000, 0, 1),
    (np.uint16, 65_536, 35_000_000_000, 0, 0), (np.uint32, 10_000, 21_000_000_000, 1, 1),
    (np.uint32, 65_536, 21_000_000_000, 0, 0), (np.uint64, 40_000, 11_000_000_000, 0, 0),
    (np.uint32, 3, 64_000_000_000, 0, 0), (np.uint32, 4, 64_000_000_000, 0, 0),
    (np.uint64, 3, 34_000_000_000, 0, 0), (np.uint64, 256, 11_000_000_000, 0, 0)])
def test_largest_builds_fit(L, dtype, sigma, n, copied, short):
    """Texts from the host that fill one GPU: text copies, planes and levels
    that are no longer needed make room for what is built next."""
    assert build_peak(L, dtype, sigma, n, copied, short) <= GPU_BYTES


def test_large_batches_build_one_size_at_a_time(L):
    """Where not all of them fit (the stand-in has no memory free), the group
    builds of a collection of more than 2^30 symbols hold the temporary memory of
    one alphabet size at a time."""
    texts = {s: [zeros((1 << 24) - 1 - i) for i in range(17)] for s in (4, 16, 64, 256)}
    before = L.fake_live()

    def build(group):
        ptr = lambda arrays: (C.c_void_p * len(arrays))(*[a.ctypes.data for a in arrays])
        al = [np.arange(s, dtype=np.uint8) for s, _ in group]
        lens = np.array([t.size for _, t in group], np.uint64)
        sigmas = np.array([s for s, _ in group], np.uint64)
        out = (C.c_void_p * len(group))()
        L.fake_reset()
        assert L.ewt_build_batch(ptr([t for _, t in group]), lens.ctypes.data, len(group), 1,
                                 ptr(al), sigmas.ctypes.data, 0, out, None) == 0
        peak, held = L.fake_peak() - before, L.fake_live() - before
        for t in out:
            assert L.ewt_free(t) == 0
        return peak, held

    alone = [build([(s, t) for t in ts]) for s, ts in texts.items()]
    peak, held = build([(s, t) for s, ts in texts.items() for t in ts])
    # (the batch grows its pool once, which the stand-in does not keep)
    assert peak <= held + max(p - h for p, h in alone)


@pytest.mark.parametrize("dtype,sigma,short,bytes_per_symbol", [
    (np.uint8, 96, 1, 5.32), (np.uint8, 129, 1, 5.32), (np.uint8, 256, 0, 5.32),
    (np.uint16, 33_024, 0, 10.62), (np.uint16, 33_024, 1, 10.62), (np.uint16, 65_536, 0, 10.62),
    (np.uint32, 10_000, 1, 21.22), (np.uint32, 65_536, 0, 21.22), (np.uint64, 40_000, 1, 42.42)])
def test_served_builds_stay_within_the_budget(L, dtype, sigma, short, bytes_per_symbol):
    """A build that the serving engine admits (its estimate is the budget, but
    for 64 MB) never holds more than the budget, also when it needs a copy of
    the text."""
    from ecl_wavelet_gb300 import serving
    for name in ("ewt_server_create", "ewt_server_destroy", "ewt_server_submit_build",
                 "ewt_server_wait"):
        f = getattr(L, name)
        f.restype, f.argtypes = serving._SIGS[name]
    size, n = np.dtype(dtype).itemsize, 4_000_000_000
    budget = int(n * bytes_per_symbol)
    cfg = serving.ServerConfig(1 << 16, 64, 1, budget, size, 0)
    server = C.c_void_p()
    assert L.ewt_server_create(0, C.byref(cfg), C.byref(server)) == 0
    text = zeros(n * size, size)  # off a 16-byte boundary
    al = np.arange(sigma, dtype=np.uint64).astype(dtype)
    bits = (sigma - 1).bit_length()
    L.fake_reset()
    for entries in {(1 << bits) + 1, sigma + 1}:
        if short:
            L.fake_patch(entries * 8, 1, 1000)
        L.fake_patch(entries * 8, (1 << bits) // 2 + 1 if short else entries - 1, n)
    before = L.fake_live()
    rid, status = C.c_uint64(), C.c_int(9)
    assert L.ewt_server_submit_build(server, text.ctypes.data, n, al.ctypes.data, sigma,
                                     C.byref(rid)) == 0
    assert L.ewt_server_wait(server, rid, C.byref(status), None, None) == 0 and status.value == 0
    peak = L.fake_peak() - before
    assert L.ewt_server_destroy(server) == 0
    assert peak <= budget


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.uint32, np.uint64])
def test_tree_bound(L, dtype):
    """EWT_MEM_TREE covers the peak of a build of every depth, from a host text
    that needs a copy, with levels that short codes leave nearly full and nearly
    empty."""
    n, size = 1 << 30, np.dtype(dtype).itemsize
    for bits in range(1, 8 * min(size, 2) + 1):
        full = 1 << bits
        for sigma, short in [(full, 0), (full // 2 + 1, 0), (full // 2 + full // 256, 1),
                             (full // 2 + full // 8 + 1, 1)]:
            if max(2, full // 2 + 1) <= sigma <= full and not (short and sigma == full):
                assert build_peak(L, dtype, sigma, n, 1, short) <= needed(L, TREE, n, size, sigma), \
                    (sigma, short)
