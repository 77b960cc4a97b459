"""What an index file holds: the tree alone, nothing of what its memory held
before, and a tag that says how its counts are to be read."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def scatter(ewt, seed):
    """Leaves the library's free memory full of other bytes."""
    rng = np.random.default_rng(seed)
    for n in (1 << 14, 1 << 17, 1 << 20, 1 << 23):
        words = rng.integers(0, 1 << 32, n // 32, dtype=np.uint64).astype(np.uint32)
        ewt.RankSelect([words], [n]).close()
        ewt.WaveletTree(rng.integers(0, 250, n // 4).astype(np.uint8)).close()


@pytest.mark.parametrize("dtype,sigma,n", [(np.uint8, 2, 50_001), (np.uint8, 5, 300_007),
                                           (np.uint8, 256, 500_001), (np.uint16, 1000, 200_003),
                                           (np.uint32, 70_000, 200_001)])
def test_same_text_same_file(ewt, tmp_path, dtype, sigma, n):
    rng = np.random.default_rng(sigma)
    text = rng.integers(0, sigma, n).astype(dtype)
    text[:sigma] = np.arange(sigma)
    files = []
    for i in range(2):
        scatter(ewt, i)
        t = ewt.WaveletTree(text, np.arange(sigma))
        t.save(str(tmp_path / str(i)))
        t.close()
        files.append((tmp_path / str(i)).read_bytes())
    assert files[0] == files[1]


def test_saved_again(ewt, tmp_path):
    """A loaded tree saves as the file that it came from, whose samples lie side
    by side; its answers and exports are the built one's."""
    rng = np.random.default_rng(1)
    text = rng.integers(0, 5, 400_001).astype(np.uint8)
    t = ewt.WaveletTree(text, np.arange(5))
    t.save(str(tmp_path / "a"))
    u = ewt.WaveletTree.load(str(tmp_path / "a"))
    u.save(str(tmp_path / "b"))
    assert (tmp_path / "a").read_bytes() == (tmp_path / "b").read_bytes()
    for l in range(t.getNumLevels()):
        for part in ("SAMPLES0", "SAMPLES1"):
            assert np.array_equal(t.export(part, l), u.export(part, l))
    batch = ewt.build_batch([text[:100_000] % 4, text % 4], [np.arange(4)] * 2)
    batch[1].save(str(tmp_path / "c"))
    v = ewt.WaveletTree.load(str(tmp_path / "c"))
    idx = rng.integers(0, text.size, 1000).astype(np.uint64)
    assert np.array_equal(v.access(idx), (text % 4)[idx])
    for l in range(2):
        for part in ("SAMPLES0", "SAMPLES1"):
            assert np.array_equal(batch[1].export(part, l), v.export(part, l))


@pytest.mark.parametrize("dtype,sigma,tag", [(np.uint8, 2, b"EWTIDX03"), (np.uint8, 256, b"EWTIDX03"),
                                             (np.uint8, 5, b"EWTIDX04"), (np.uint16, 1000, b"EWTIDX04"),
                                             (np.uint32, 70_000, b"EWTIDX03")])
def test_tags(ewt, tmp_path, dtype, sigma, tag):
    """Group levels over padded codes have a tag of their own, which readers of
    the older form refuse; the older tag before such levels is still read."""
    rng = np.random.default_rng(sigma)
    text = rng.integers(0, sigma, 150_001).astype(dtype)
    text[:sigma] = np.arange(sigma)
    t = ewt.WaveletTree(text, np.arange(sigma))
    t.save(str(tmp_path / "i"))
    raw = (tmp_path / "i").read_bytes()
    assert raw[:8] == tag
    idx = rng.integers(0, text.size, 1000).astype(np.uint64)
    for magic in (tag, b"EWTIDX03"):
        (tmp_path / "j").write_bytes(magic + raw[8:])
        u = ewt.WaveletTree.load(str(tmp_path / "j"))
        assert np.array_equal(u.access(idx), text[idx])
    (tmp_path / "j").write_bytes(b"EWTIDX05" + raw[8:])
    with pytest.raises(ewt.EwtError):
        ewt.WaveletTree.load(str(tmp_path / "j"))
