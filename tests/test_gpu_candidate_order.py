"""Candidate ranking and placement at their limits (gpu): more candidates in one
band than are ranked from shared memory, candidates past the cap, frames of one
band and of the most bands, against the oracle's candidate list.
"""
import numpy as np
import pytest

import bdcudatag
import oracle
from gpu_checks import check_frame

pytestmark = pytest.mark.gpu


def boxes(width, height, step, size=6, rows=None):
    """Hollow dark squares on white, `step` pixels apart: each a candidate."""
    img = np.full((height, width), 220, np.uint8)
    ys = range(8, height - size - 2, step) if rows is None else rows
    for y in ys:
        for x in range(8, width - size - 2, step):
            img[y:y + size, x:x + size] = 30
            img[y + 2:y + size - 2, x + 2:x + size - 2] = 220
    return img


@pytest.mark.parametrize("width,height,step,rows", [
    (8192, 32, 9, [9]),          # 900 candidates in one band: past the 512 of shared memory
    (4096, 48, 9, [9, 18]),      # 450 a band
    (640, 480, 8, None),         # 4,500 in the frame: past the cap
    (64, 16, 9, [8]),            # two bands
    (32, 16384, 20, None),       # the most bands
])
def test_candidates(width, height, step, rows):
    img = boxes(width, height, step, rows=rows)
    cfg = dict(min_tag_pixels=4, min_cluster_pixels=4)
    check_frame(img, 1, bdcudatag.default_config(**cfg), oracle.default_config(**cfg))
