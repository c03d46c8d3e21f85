"""Device memory that a graph build leaves reserved in the engine's pool."""
import pytest

import indigo2suite_b200 as i2

pytestmark = pytest.mark.gpu


def test_a_build_keeps_at_most_its_pooled_scratch(gpu):
    import torch

    free = lambda: torch.cuda.mem_get_info()[0]
    i2.DeviceGraph.generate_er(1000, 4000, seed=1).free()  # contexts, kernels, the pool itself
    i2.trim_device_memory()
    before = free()
    # candidate pairs of 1.0 GB a buffer beside the 0.96 GB of kept pairs
    i2.DeviceGraph.generate_er(1 << 20, 120_000_000, seed=2, weighted=False).free()
    kept = before - free()
    i2.trim_device_memory()
    # 2 GB of scratch; the graph's own arrays (0.96 GB) take the place of freed scratch
    assert kept <= (2 << 30) + (256 << 20), kept
    assert before - free() <= 64 << 20
