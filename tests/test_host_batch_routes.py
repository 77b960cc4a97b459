"""Which way a host batch takes (over the stand-in runtime, tests/fake_cuda): one
type of query is answered in place up to 2^21 queries, unless its results have 8
MiB and more of pages to be populated; mixed batches are copied chunk by chunk
from 2^19 queries on."""
import mmap

import numpy as np
import pytest

from tests import fake_cuda

LOW, HIGH = 1 << 19, 1 << 21


@pytest.fixture(scope="module")
def setup():
    L = fake_cuda.load()
    L.fake_set(b"host_type", 0)  # memory that CUDA knows nothing of
    tree = fake_cuda.build(L, np.zeros(1000, np.uint8), np.arange(2, dtype=np.uint8))
    yield L, tree
    L.ewt_free(tree)


@pytest.mark.parametrize("m,kind,fresh,copied", [
    (LOW - 1, "mixed", 0, False), (LOW - 1, "rank", 1, False), (LOW, "mixed", 0, True),
    (LOW, "rank", 0, False), (LOW, "access", 0, False), (HIGH // 2 - 1, "rank", 1, False),
    (HIGH // 2, "rank", 1, True), (HIGH // 2, "rank", 0, False), (HIGH - 1, "select", 0, False),
    (HIGH - 1, "access", 1, False), (HIGH, "rank", 0, True)])
def test_route(setup, m, kind, fresh, copied):
    L, tree = setup
    types, q = np.zeros(m, np.uint8), np.zeros((m, 2), np.uint64)
    nbytes = m * (1 if kind == "access" else 8)
    out = np.frombuffer(mmap.mmap(-1, nbytes), np.uint8)
    if not fresh:
        out[:] = 1
    L.fake_reset()
    st = {"mixed": lambda: L.ewt_mixed(tree, types.ctypes.data, q.ctypes.data, m, out.ctypes.data),
          "rank": lambda: L.ewt_rank(tree, q.ctypes.data, m, out.ctypes.data),
          "select": lambda: L.ewt_select(tree, q.ctypes.data, m, out.ctypes.data),
          "access": lambda: L.ewt_access(tree, q.ctypes.data, m, out.ctypes.data)}[kind]()
    assert st == 0
    assert ("copy_kernel" in L.fake_journal().decode()) == copied
