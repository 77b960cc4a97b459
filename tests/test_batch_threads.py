"""ewt_build_batch on a system that gives it fewer threads than it asks for
(over the stand-in runtime, tests/fake_cuda): the batch is built all the same,
where an exception out of a thread's start would end the process."""
import subprocess
import sys

import pytest

from tests.conftest import REPO

SCRIPT = """
import ctypes as C, sys
import numpy as np
sys.path.insert(0, %r)
from tests import fake_cuda
L = fake_cuda.load()
texts = [np.zeros(100 + i, np.uint8) for i in range(9)]
sigmas = np.array([4, 16, 64, 2, 2, 2, 4, 16, 64], np.uint64)
al = [np.arange(s, dtype=np.uint8) for s in sigmas]
lens = np.array([t.size for t in texts], np.uint64)
ptr = lambda arrays: (C.c_void_p * len(arrays))(*[a.ctypes.data for a in arrays])
out, st = (C.c_void_p * 9)(), np.full(9, 7, np.int32)
L.fake_reset()
L.fake_fail(b"thread", %d)
rc = L.ewt_build_batch(ptr(texts), lens.ctypes.data, 9, 1, ptr(al), sigmas.ctypes.data, 0, out,
                       st.ctypes.data)
assert rc == 0, L.ewt_last_error()
assert (st == 0).all() and all(out), (st, list(out))
"""


@pytest.mark.parametrize("nth", range(1, 7))
def test_a_thread_is_refused(nth):
    from tests import fake_cuda
    fake_cuda.load()
    r = subprocess.run([sys.executable, "-c", SCRIPT % (REPO, nth)], capture_output=True, text=True,
                       timeout=120)
    assert r.returncode == 0, (r.returncode, r.stderr[-2000:])
