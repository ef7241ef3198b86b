"""The bench names the pair kernel that ran (CPU test of its labels)."""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

import bench  # noqa: E402


def test_kernel_label_follows_the_launches():
    shape = {"threads": 384, "ipt": 1, "tile": 512}
    assert bench.kernel_that_ran(3.0, shape) == {"kernel": "k_newton", "threads": 128, "ipt": 8, "tile": 32}
    assert bench.kernel_that_ran(2.0, shape) == dict(shape, kernel="k_pairs_mixed_fused")
    assert bench.flops_per_pair(3.0) < bench.flops_per_pair(2.0)
