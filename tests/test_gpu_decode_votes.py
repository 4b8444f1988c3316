"""Quads whose four rotations part ways in the decoder (gpu): a contrast within
rounding of the limit is above it in one rotation and below it in another, so
some rotations go on to the border test and others do not.  The kernels return
and give the oracle's result at every stage.
"""
import pytest

import bdcudatag
import oracle
import scenes
from gpu_checks import check_frame, same_records

pytestmark = pytest.mark.gpu

# (scene set, frame index, width, height): noisy frames that hold such a quad.
FRAMES = [
    (scenes.EIGHT_TAGS_640, 478, 640, 480),
    (scenes.MULTI_SIZE, 233, 1283, 717),
    (scenes.MULTI_SIZE, 435, 1280, 800),
    (scenes.MULTI_SIZE, 66, 1920, 1080),
    (scenes.SERVING, 22, 1920, 1080),
    (scenes.SERVING, 46, 3840, 2160),
]


@pytest.mark.parametrize("scene,index,width,height", FRAMES)
def test_rotations_at_the_contrast_limit(scene, index, width, height):
    img, _ = scenes.render_scene(scene, index, width, height)
    for family in (0, 1):
        check_frame(img, family)


@pytest.mark.parametrize("split", [0, 32])
def test_both_fit_paths(split):
    """As a batch, every candidate by a warp (split 0) or the larger ones by
    a CTA.  The last frame is the one that showed the fault."""
    frames = [scenes.render_scene(s, i, w, h)[0] for s, i, w, h in FRAMES[1:4]]
    frames.append(scenes.render_scene(scenes.MULTI_SIZE, 3, 1920, 1080,
                                      seed=1_000_000 + 4096 * 253228486 + 3)[0])
    batch = bdcudatag.Batch([(f.shape[1], f.shape[0], 3) for f in frames])
    batch.set_launch(quad_split=split)
    found, out = batch.detect(frames)
    for k, f in enumerate(frames):
        for family in (0, 1):
            n, want = oracle.Frame(f, family).detections()
            assert found[k, family] == n
            same_records(out[k, family, :n], want)
