"""The bit-plane passes of the build (planes.cuh) where their bookkeeping can
go wrong: texts ending at the edges of a tile (a CTA's slots of 128 symbols,
less the slots that class runs may waste), for every pass plan; texts whose
runs are all zeros, all ones, sorted or alternate, so that slots hold only one
child's symbols and runs start at every bit offset; symbols mapped to codes on
the way in.  Integer results: byte-identical to the oracle's."""
import numpy as np
import pytest

from tests.test_gpu_parity import assert_same_tree, check_queries

pytestmark = pytest.mark.gpu


def tile(slots, k):
    return (slots - ((5 << k) + 3) // 4) * 128


# code bits -> slots and levels of the first pass
FIRST = {1: (256, 0), 2: (256, 1), 3: (256, 2), 4: (256, 3), 5: (256, 4), 8: (256, 3),
         9: (256, 4), 10: (128, 3), 16: (128, 3)}


def same(ewt, oracle, text, alphabet, seed=1):
    gt = ewt.WaveletTree(text, alphabet)
    ot = oracle.OracleTree(text, alphabet)
    assert_same_tree(gt, ot)
    check_queries(gt, ot, text, np.asarray(alphabet, dtype=np.uint64), 1_000, seed=seed)


@pytest.mark.parametrize("L", sorted(FIRST))
@pytest.mark.parametrize("tiles,more", [(1, -1), (1, 0), (1, 1), (2, 127), (3, 33)])
def test_tile_edges(ewt, oracle, L, tiles, more):
    n = tiles * tile(*FIRST[L]) + more
    dtype = np.uint8 if L <= 8 else np.uint16
    rng = np.random.default_rng(1000 * L + tiles + more)
    text = rng.integers(0, 1 << L, n, dtype=np.uint64).astype(dtype)
    same(ewt, oracle, text, np.arange(1 << L))


@pytest.mark.parametrize("shape", ["zeros", "ones", "sorted", "blocks", "rare"])
@pytest.mark.parametrize("L", [5, 8, 12])
def test_one_sided_slots(ewt, oracle, L, shape):
    n, sigma = 70_001, 1 << L
    dtype = np.uint8 if L <= 8 else np.uint16
    rng = np.random.default_rng(L)
    text = {"zeros": np.zeros(n, np.int64), "ones": np.full(n, sigma - 1),
            "sorted": np.sort(rng.integers(0, sigma, n)),
            "blocks": np.repeat(rng.integers(0, sigma, n // 37 + 1), 37)[:n],
            "rare": np.where(rng.random(n) < 0.001, rng.integers(0, sigma, n), sigma // 2)}[shape]
    same(ewt, oracle, text.astype(dtype), np.arange(sigma))


@pytest.mark.parametrize("dtype,sigma", [(np.uint8, 2), (np.uint8, 64), (np.uint16, 512)])
def test_mapped_symbols(ewt, oracle, dtype, sigma):
    """Scattered alphabets of a power of two, detected from the text."""
    rng = np.random.default_rng(sigma)
    alphabet = np.sort(rng.choice(np.iinfo(dtype).max, sigma, replace=False)).astype(dtype)
    text = alphabet[rng.integers(0, sigma, 50_021)]
    text[:sigma] = alphabet
    same(ewt, oracle, text, alphabet)
    assert np.array_equal(ewt.WaveletTree(text).export("COUNTS"),
                          ewt.WaveletTree(text, alphabet).export("COUNTS"))
    if alphabet[-1] < np.iinfo(dtype).max:
        bad = text.copy()
        bad[-1] = np.iinfo(dtype).max
        with pytest.raises(ewt.EwtError):
            ewt.WaveletTree(bad, alphabet)


@pytest.mark.parametrize("dtype,sigma", [(np.uint8, 3), (np.uint8, 5), (np.uint8, 129),
                                         (np.uint8, 255), (np.uint16, 257), (np.uint16, 1000),
                                         (np.uint16, 40_001), (np.uint32, 300),
                                         (np.uint32, 4096), (np.uint64, 5000)])
@pytest.mark.parametrize("skew", ["uniform", "first", "last"])
def test_short_codes(ewt, oracle, dtype, sigma, skew):
    """Alphabets with short codes (their padding ends the levels) and wide
    symbols, scattered and detected; texts dominated by the first (longest
    code) or the last symbol (shortest: levels mostly empty, packed)."""
    rng = np.random.default_rng(sigma)
    top = min(np.iinfo(dtype).max, 1 << 62)
    alphabet = np.sort(rng.choice(top, sigma, replace=False) if top < 1 << 17 else
                       np.unique(rng.integers(0, top, 2 * sigma + 10))[:sigma]).astype(dtype)
    n = max(61_003, 2 * sigma)
    ids = rng.integers(0, sigma, n)
    if skew != "uniform":
        ids = np.where(rng.random(n) < 0.03, ids, 0 if skew == "first" else sigma - 1)
    ids[rng.permutation(n)[:sigma]] = np.arange(sigma)
    text = alphabet[ids]
    same(ewt, oracle, text, alphabet)
    detected = ewt.WaveletTree(text)
    assert np.array_equal(detected.getAlphabet(), alphabet)
    assert np.array_equal(detected.export("LEVEL_WORDS", 1),
                          ewt.WaveletTree(text, alphabet).export("LEVEL_WORDS", 1))


@pytest.mark.parametrize("n", [1, 2, 31, 33, 13_823, 13_824, 13_825, 30_208 + 1])
def test_short_codes_edges(ewt, oracle, n):
    """Given minimal alphabets of no power of two; every code length present
    (the last symbol of each length is appended)."""
    for dtype, sigma in ((np.uint8, 75), (np.uint16, 2300)):
        rng = np.random.default_rng(n + sigma)
        text = np.concatenate([rng.integers(0, sigma, n), np.arange(sigma)]).astype(dtype)
        same(ewt, oracle, text, np.arange(sigma))


@pytest.mark.parametrize("sigma", [5, 75, 200])
@pytest.mark.parametrize("n", [43, 21_503, 21_505, 2 * 49_152 + 95])
def test_padded_group_levels(ewt, oracle, sigma, n, tmp_path):
    """Group query levels over padded codes at their superblock boundaries
    (21,504 octal, 49,152 quad digits); again from an index file, and at other
    select-sample rates."""
    rng = np.random.default_rng(n + sigma)
    alphabet = np.arange(sigma)
    text = rng.integers(0, sigma, max(n, sigma)).astype(np.uint8)
    text[rng.permutation(text.size)[:sigma]] = np.arange(sigma)
    gt = ewt.WaveletTree(text, alphabet)
    ot = oracle.OracleTree(text, alphabet)
    al = alphabet.astype(np.uint64)
    check_queries(gt, ot, text, al, 1_000, seed=n)
    gt.save(str(tmp_path / "i"))
    lt = ewt.WaveletTree.load(str(tmp_path / "i"))
    check_queries(lt, ot, text, al, 1_000, seed=n + 1)
    for rate in (0, 1024):
        gt.set_select_samples(rate)
        check_queries(gt, ot, text, al, 1_000, seed=rate)


@pytest.mark.parametrize("dtype,kind", [(np.uint32, "dense"), (np.uint32, "clustered"),
                                        (np.uint64, "clustered"), (np.uint64, "two"),
                                        (np.uint32, "large"), (np.uint64, "shared")])
def test_wide_alphabets(ewt, oracle, dtype, kind):
    """Detection and search of 4- and 8-byte alphabets: consecutive symbols; all
    but one in one bucket of the search's range; two symbols at the type's
    ends; more symbols than are searched in shared memory, and than are sorted
    on the device."""
    rng = np.random.default_rng(7)
    top = int(np.iinfo(dtype).max)
    a = {"dense": np.arange(1000, 1900), "clustered": np.append(np.arange(5, 3005, 3), top),
         "two": np.array([0, top], dtype=np.uint64), "shared": np.arange(20_000) * (top // 20_001),
         "large": np.arange(70_000) * 61_001}[kind].astype(dtype)
    text = a[rng.integers(0, a.size, max(100_001, 2 * a.size))]
    text[:a.size] = a
    same(ewt, oracle, text, a)
    assert np.array_equal(ewt.WaveletTree(text).getAlphabet(), a)
    if a[0] > 0:  # a symbol below all others stands for the first
        below = text.copy()
        below[-1] = 0
        gt, ot = ewt.WaveletTree(below, a), ewt.WaveletTree(np.append(text[:-1], a[:1]), a)
        assert np.array_equal(gt.export("COUNTS"), ot.export("COUNTS"))
