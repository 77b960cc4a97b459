"""The bench's model of the bit-plane passes, which its roofline divides by:
the pass plan, a hand-kept mirror of plan_plane_passes (planes.cuh), against the
passes that the library launches (over the stand-in runtime, tests/fake_cuda),
and the bytes of a pass against counts by hand."""
import numpy as np
import pytest

import bench
from tests import fake_cuda


@pytest.mark.parametrize("L", range(1, 17))
def test_plan(L):
    plan = bench.plane_pass_plan(L)
    assert sum(plan) == L - 1 and all(1 <= k <= 4 for k in plan)
    lib = fake_cuda.load()
    n = 100_000
    dtype = np.uint8 if L <= 8 else np.uint16
    tree = fake_cuda.build(lib, np.zeros(n, dtype),
                           np.arange(1 << L, dtype=np.uint64).astype(dtype),
                           ((1 << L) + 1, 1 << L, n))
    lines = [x.split() for x in lib.fake_journal().decode().splitlines()]
    lib.ewt_free(tree)
    passes = [x for x in lines if "plane_pass_kernel" in x[0]]
    assert len(passes) == len(plan)
    # a pass from level a carries the L - 1 - a planes behind level a's: two
    # buffers of 4-word slots and pads each (planes.cuh pass_smem)
    a = 0
    for k, (_, _, block, smem) in zip(plan, passes):
        slots = int(block)
        assert int(smem) == 2 * 4 * ((L - 1 - a) * (4 * slots + 8) + 8)
        a += k


def test_bytes_per_launch():
    n = 1 << 30
    # 256 symbols (levels 1-3, then 4-7; group levels at 0, 3, 6): 8 planes in,
    # levels 1-3 and the 4 deeper planes of the level-3 order out; 5 in, levels
    # 4-7 and 1 deeper plane of the level-6 order out
    assert bench.plane_pass_bytes_per_launch(n, 8) == (15 + 10) * n / 8 / 2
    # 16 symbols (levels 1-3; group levels at 0, 2): 4 in, 3 and 1 of level 2 out
    assert bench.plane_pass_bytes_per_launch(n, 4) == 8 * n / 8
    # 4 symbols (level 1, group level at 0): 2 in, 1 out
    assert bench.plane_pass_bytes_per_launch(n, 2) == 3 * n / 8
    # 65,536 symbols (1-3, 4-7, 8-11, 12-15; group levels at 0, 3, 6, 9, 12, 14):
    # 16 in, 3 + 12 out; 13 in, 4 + 8 and 2 of level 6 out; 9 in, 4 + 4 and 2 of
    # level 9 out; 5 in, 4 and 1 each of levels 12 and 14 out
    assert bench.plane_pass_bytes_per_launch(n, 16) == (31 + 27 + 19 + 11) * n / 8 / 4
    assert bench.plane_pass_bytes_per_launch(n, 1) == 0.0
