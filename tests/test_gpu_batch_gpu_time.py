"""The GPU time of a batch of pageable frames does not count the CPU's work (gpu).

Eight frames of 1283x717 with a gap between their rows are compacted by the CPU, for
several hundred microseconds; the same frames without a gap are not.  Both are then copied
to the device.  The copies of 7.4 MB take under 100 us either way, so the GPU times
differ by less than that; the least of many calls of each.
"""
import numpy as np
import pytest

import bdcudatag
import scenes

pytestmark = pytest.mark.gpu

W, H, N = 1283, 717, 8


def test_gpu_time():
    frames = [np.ascontiguousarray(f) for f in scenes.ref_scenes(W, H, N)[0]]
    gapped = []
    for f in frames:
        rows = np.zeros((H, W + 5), np.uint8)
        rows[:, :W] = f
        gapped.append(rows)
    batch = bdcudatag.Batch([(W, H, 1)] * N)
    times = {}
    for name, rows in (("tight", frames), ("gapped", gapped)):
        times[name] = []
        for _ in range(30):
            batch.detect(rows)
            times[name].append(batch.last_gpu_ms())
    assert min(times["gapped"]) < min(times["tight"]) + 0.1, {k: min(v) for k, v in times.items()}
