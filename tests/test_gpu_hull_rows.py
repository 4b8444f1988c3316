"""Boundary rows of a candidate at the words' edges (gpu): rings whose sides lie on,
before and after a multiple of 32 px, in rows full of other runs, and rings of more
rows than are kept, against the oracle at every stage.
"""
import numpy as np
import pytest

from gpu_checks import check_frame

pytestmark = pytest.mark.gpu


def ring(img, x0, y0, x1, y1, width):
    img[y0:y1 + 1, x0:x1 + 1] = 30
    img[y0 + width:y1 + 1 - width, x0 + width:x1 + 1 - width] = 220


@pytest.mark.parametrize("left,right", [(31, 64), (32, 63), (32, 95), (33, 96), (30, 31 + 64), (64, 65 + 30), (1, 62)])
@pytest.mark.parametrize("stripes", [0, 2, 3])
def test_word_edges(left, right, stripes):
    img = np.full((96, 160), 220, np.uint8)
    ring(img, left, 20, right, 70, 4)
    if stripes:  # runs inside and beside the ring, every few pixels
        for x in list(range(left + 6, right - 6, stripes)) + list(range(right + 4, 156, stripes)):
            img[30:60, x] = 30
    check_frame(img, 0)
    check_frame(img, 1)


@pytest.mark.parametrize("rows", [1024, 1025, 1300])
def test_more_rows_than_kept(rows):
    img = np.full((rows + 40, 700), 220, np.uint8)
    ring(img, 40, 20, 340, 19 + rows, 60)
    img[300:340, 0:20] = 30
    check_frame(img, 0)
