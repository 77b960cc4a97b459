"""Large host batches, whose queries and results are copied by kernels chunk by
chunk: sizes around the threshold and with ragged last chunks, every record
size, buffers at odd addresses.  The answers are those of small batches, which
are answered in place (and are compared with the oracle elsewhere)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MIN = 1 << 19  # queries from which batches are copied in chunks


@pytest.fixture(scope="module")
def tree(ewt):
    rng = np.random.default_rng(3)
    text = rng.integers(0, 75, 300_007).astype(np.uint8)
    return text, ewt.WaveletTree(text, np.arange(75))


@pytest.mark.parametrize("m", [MIN - 1, MIN, MIN + 1, MIN + (1 << 17) + 15, 5 * (MIN // 4) + 3])
def test_sizes(tree, m):
    text, t = tree
    rng = np.random.default_rng(m)
    types = rng.integers(0, 3, m).astype(np.uint8)
    q = t.make_queries(rng.integers(1, text.size // 100, m), rng.integers(0, 75, m))
    got = t.mixed(types, q)
    step = 100_000
    want = np.concatenate([t.mixed(types[a:a + step], q[a:a + step]) for a in range(0, m, step)])
    assert np.array_equal(got, want)
    idx = rng.integers(0, text.size, m).astype(np.uint64)
    assert np.array_equal(t.access(idx), text[idx.astype(np.int64)])


@pytest.mark.parametrize("shift", [0, 1, 4, 8])
def test_odd_addresses(ewt, tree, shift):
    text, t = tree
    m = 4 * MIN + 77  # shorter batches want 8-byte aligned queries
    rng = np.random.default_rng(shift)
    idx = rng.integers(0, text.size, m).astype(np.uint64)
    room_in, room_out = np.zeros(m * 8 + 32, np.uint8), np.zeros(m + 16, np.uint8)
    a = (-room_in.ctypes.data) % 16 + shift
    room_in[a:a + m * 8] = idx.view(np.uint8)
    b = shift if shift else 3
    assert ewt.lib().ewt_access(t.handle, room_in.ctypes.data + a, m, room_out.ctypes.data + b) == 0
    assert np.array_equal(room_out[b:b + m], text[idx.astype(np.int64)])
    assert not room_out[:b].any() and not room_out[b + m:].any()


@pytest.mark.parametrize("m", [MIN + 7, 4 * MIN + 33])
@pytest.mark.parametrize("pinned", [(True, True), (True, False), (False, True)])
def test_pinned_buffers(ewt, tree, m, pinned):
    torch = pytest.importorskip("torch")
    text, t = tree
    rng = np.random.default_rng(m)

    def room(count, dtype, pin):
        return torch.zeros(count * dtype().itemsize, dtype=torch.uint8, pin_memory=pin).numpy().view(dtype)

    idx, out = room(m, np.uint64, pinned[0]), room(m, np.uint8, pinned[1])
    idx[:] = rng.integers(0, text.size, m)
    assert ewt.lib().ewt_access(t.handle, idx.ctypes.data, m, out.ctypes.data) == 0
    assert np.array_equal(out, text[idx.astype(np.int64)])
