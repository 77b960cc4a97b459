"""Mixed batches over an index of more than 1 GiB of level bits, whose query
types are walked list by list: batch sizes and mixes at the edges of warps and
chunks give the answers of the calls for one type (compared with the oracle
and the plain scan elsewhere)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tree(ewt):
    torch = pytest.importorskip("torch")
    n = (1 << 32) + 77
    gen = torch.Generator(device="cuda").manual_seed(5)
    text = torch.empty(n, dtype=torch.uint8, device="cuda").random_(0, 4, generator=gen)
    torch.cuda.synchronize()
    t = ewt.WaveletTree(text, np.arange(4))
    yield n, t
    t.close()


@pytest.mark.parametrize("m", [1, 31, 65, 257, 70_001])
@pytest.mark.parametrize("mix", [(1, 1, 1), (0, 0, 1), (8, 0, 1), (0, 9, 1), (1, 0, 0)])
def test_mixes(tree, m, mix):
    n, t = tree
    rng = np.random.default_rng(m)
    types = rng.choice(3, m, p=np.array(mix) / sum(mix)).astype(np.uint8)
    index = np.where(types == 2, rng.integers(1, n // 5, m), rng.integers(0, n, m))
    q = t.make_queries(index, rng.integers(0, 4, m))
    want = np.zeros(m, np.uint64)
    a, r, s = (types == k for k in range(3))
    if a.any():
        want[a] = t.access(q["index"][a])
    if r.any():
        want[r] = t.rank(q[r])
    if s.any():
        want[s] = t.select(q[s])
    assert np.array_equal(t.mixed(types, q), want)
