"""The bit-plane passes are launched as one wave of CTAs: every CTA of a pass
fits at once beside the others by shared memory (228 KB per SM; over the
stand-in runtime, which answers the occupancy query from it, tests/fake_cuda).
Sizes: every number of carried planes."""
import numpy as np
import pytest

from tests import fake_cuda

SMS, STATIC, RESERVED = 152, 1584, 1024


@pytest.mark.parametrize("L", range(2, 17))
def test_one_wave(L):
    lib = fake_cuda.load()
    lib.fake_set(b"static_smem", STATIC)
    n = 40_000_000
    dtype = np.uint8 if L <= 8 else np.uint16
    tree = fake_cuda.build(lib, np.zeros(n, dtype), np.arange(1 << L, dtype=np.uint64).astype(dtype),
                           ((1 << L) + 1, 1 << L, n))
    passes = [list(map(int, x.split()[1:])) for x in lib.fake_journal().decode().splitlines()
              if "plane_pass_kernel" in x]
    lib.ewt_free(tree)
    assert passes
    for grid, block, smem in passes:
        fit = (228 << 10) // (smem + STATIC + RESERVED)
        assert grid <= SMS * fit, (grid, block, smem)
        # ... and the GPU is full: there are more chunks than CTAs
        assert grid >= SMS * min(fit, 3)


@pytest.mark.parametrize("fit", [7, 10, 16])
def test_one_wave_of_counts(fit):
    """The digit counts of a later pass, too, whatever number of CTAs fits."""
    lib = fake_cuda.load()
    lib.fake_set(b"max_ctas", fit)
    n = 100_000_000
    tree = fake_cuda.build(lib, np.zeros(n, np.uint8), np.arange(256, dtype=np.uint8), (257, 256, n))
    lib.fake_set(b"max_ctas", 32)
    grids = [int(x.split()[1]) for x in lib.fake_journal().decode().splitlines()
             if "plane_counts_kernel" in x]
    lib.ewt_free(tree)
    assert grids == [SMS * fit]
