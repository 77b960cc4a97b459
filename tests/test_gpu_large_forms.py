"""The paths of builds and batches that only large sizes take."""
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_passes_of_the_largest_texts(ewt):
    """64-bit word indices (texts of 2^36 symbols), orders in two allocations (of
    more than 32 GB) and texts read in parts (codes of more than 32 GB), at small
    sizes: the same levels, class starts and kept planes as the usual form's."""
    from ecl_wavelet_gb300 import dropin
    r = subprocess.run([dropin.build_example("plane_limits"), "7"], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    lines = r.stdout.splitlines()
    assert len(lines) == 56 and all(l.endswith(": 0 differences") for l in lines), r.stdout


@pytest.mark.parametrize("sigma,short", [(96, 0), (96, 1), (5, 1)])
def test_short_codes_over_many_tiles(ewt, oracle, sigma, short):
    """An alphabet of no power of two over more than 2,048 tiles (the scan in
    three launches), with levels that stay where the passes put them and with
    levels that are packed: exports and answers are the oracle's."""
    from tests.test_gpu_fullsize import LEVEL_PARTS, TREE_PARTS
    from tests.workloads import mixed_queries_from_counts
    n = 2_200 * 31_488 + 77
    rng = np.random.default_rng(sigma + short)
    text = rng.integers(0, sigma, n, dtype=np.uint8)
    if short:  # mostly the symbol of the shortest code
        text[rng.random(n, dtype=np.float32) < 0.95] = sigma - 1
    al = np.arange(sigma, dtype=np.uint64)
    gt = ewt.WaveletTree(text, al)
    ot = oracle.OracleTree(text, al, threads=0)
    for p in TREE_PARTS:
        assert np.array_equal(gt.export(p), ot.export(p)), p
    for l in range(gt.getNumLevels()):
        for p in LEVEL_PARTS:
            assert np.array_equal(gt.export(p, l), ot.export(p, l)), (p, l)
    occ = np.diff(np.append(gt.export("COUNTS").astype(np.int64), n))
    types, index, sym = mixed_queries_from_counts(rng, n, occ, 1 << 20)
    want, st = oracle.scan_batch(text, sigma, types, index, sym)
    assert st == 0
    assert np.array_equal(gt.mixed(types, gt.make_queries(index, sym)), want)
    gt.close()


@pytest.fixture(scope="module")
def large_tree(ewt):
    torch = pytest.importorskip("torch")
    n = (1 << 32) + 77
    gen = torch.Generator(device="cuda").manual_seed(5)
    text = torch.empty(n, dtype=torch.uint8, device="cuda").random_(0, 4, generator=gen)
    torch.cuda.synchronize()
    t = ewt.WaveletTree(text, np.arange(4))
    yield n, t
    t.close()


@pytest.mark.parametrize("mix", [(1, 1, 1), (0, 0, 1), (8, 0, 1), (0, 9, 1), (1, 0, 0), (300, 1, 1)])
def test_full_chunks_list_by_list(large_tree, mix):
    """Mixed batches over an index of more than 1 GiB, in chunks of 2,048: lists
    of several rounds of a CTA's threads, begun on any of its warps.  The
    answers are those of the calls for one type."""
    n, t = large_tree
    m = 152 * 8 * 2048 + 1  # at least as many as fill the chunks of all CTAs
    rng = np.random.default_rng(sum(mix))
    types = rng.choice(3, m, p=np.array(mix) / sum(mix)).astype(np.uint8)
    index = np.where(types == 2, rng.integers(1, n // 5, m), rng.integers(0, n, m))
    q = t.make_queries(index, rng.integers(0, 4, m))
    want = np.zeros(m, np.uint64)
    for k, call in enumerate((lambda x: t.access(x["index"]), t.rank, t.select)):
        if (types == k).any():
            want[types == k] = call(q[types == k])
    assert np.array_equal(t.mixed(types, q), want)


def test_symbol_at_the_end_of_the_type(ewt, oracle):
    """A 64-bit alphabet whose last symbol is 2^64 - 1, which marks an empty slot
    of the set of distinct symbols."""
    from tests.test_gpu_planes import same
    al = np.append(np.arange(5, 3005, 3, dtype=np.uint64), np.uint64(2**64 - 1))
    assert int(al[-1]) == 2**64 - 1
    text = al[np.random.default_rng(7).integers(0, al.size, 100_001)]
    text[:al.size] = al
    same(ewt, oracle, text, al)
    assert np.array_equal(ewt.WaveletTree(text).getAlphabet(), al)
