"""Host-side facts that bench.py states about the calls it times."""
import pytest

import bench


@pytest.mark.parametrize("n,split", [(1, False), ((1 << 21) - 1, False), (1 << 21, True),
                                     (16 * 4096 * 4096, True), (531_678_720, True),
                                     (531_678_721, False), (1 << 30, False)])
def test_two_map_kernels_between_the_limits(n, split):
    assert bench.splits_u32_map(n) == split
