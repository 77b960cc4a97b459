"""Detection of 4- and 8-byte alphabets of more symbols than the first hash set
holds (which is then made larger, and the text read again)."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,sigma", [(np.uint32, 32_768), (np.uint32, 32_769),
                                         (np.uint64, 66_000), (np.uint32, 1_000_000)])
def test_many_symbols(ewt, dtype, sigma):
    """The symbols are those of the text, and finding them costs a few reads of
    the text and a sort of the symbols, not a walk around the full set per
    symbol (of a million symbols: 0.1 against 20 s)."""
    rng = np.random.default_rng(sigma)
    al = np.unique(rng.integers(0, np.iinfo(dtype).max, sigma + sigma // 8, dtype=dtype))
    al = np.sort(rng.permutation(al)[:sigma])
    text = al[rng.integers(0, sigma, 20_000_000)]
    text[rng.permutation(text.size)[:sigma]] = al
    ewt.WaveletTree(text[:100_000].copy()).close()
    t0 = time.perf_counter()
    t = ewt.WaveletTree(text, al)
    given = time.perf_counter() - t0
    t.close()
    t0 = time.perf_counter()
    t = ewt.WaveletTree(text)
    detected = time.perf_counter() - t0
    assert np.array_equal(t.getAlphabet(), al)
    t.close()
    assert detected < given + 1.0, (detected, given)
