"""Batches over many trees, cut into work items whose size follows the batch:
sizes around one item, one item per tree and the largest items; the answers
are those that every tree gives by itself (compared with the oracle
elsewhere)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 255, 257, 3 * 256 + 31, 160_001, 1_300_003])
@pytest.mark.parametrize("kinds", [(0, 1, 2), (2,), (0, 2)])
def test_item_sizes(ewt, m, kinds):
    rng = np.random.default_rng(m)
    texts = [rng.integers(0, s, n).astype(np.uint8) for n, s in [(5000, 256), (70_001, 16), (333, 75)]]
    trees = ewt.build_batch(texts, [np.arange(256), np.arange(16), np.arange(75)])
    which = np.sort(rng.integers(0, 3, m)).astype(np.uint32)
    types = rng.choice(kinds, m).astype(np.uint8)
    q = trees[0].make_queries(rng.integers(1, 300, m), rng.integers(0, 16, m))
    want = np.concatenate([t.mixed(types[which == i], q[which == i])
                           for i, t in enumerate(trees) if (which == i).any()])
    order = rng.permutation(m)
    got = ewt.mixed_multi(trees, which[order], types[order], q[order])
    assert np.array_equal(got, want[order])
