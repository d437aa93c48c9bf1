"""The benchmark's roofline line names the lidar kernel that its shape runs."""
import sys
from pathlib import Path

import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))
import bench  # noqa: E402


@pytest.mark.parametrize("flat,dynamic,kernel", [(0, 0, "k_lidar_track"), (1, 0, "k_lidar_flat"),
                                                 (0, 1, "k_lidar_dynamic")])
def test_lidar_kernel(flat, dynamic, kernel):
    assert bench.lidar_kernel({"cars_per_block": 2, "wide": 0, "split": 0, "dynamic": dynamic, "order": [0],
                               "flat": flat}) == kernel
