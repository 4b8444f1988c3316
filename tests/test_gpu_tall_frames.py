"""Candidate tables of tall frames (gpu): in shared memory up to 1,024 bands, in global
memory beyond.  Frames at and around the bound, alone, in a batch of several heights and
by the persistent launch, against the oracle's candidate list; and the time of four tall frames
against one: they share the GPU, and what their CTAs ask of an SM must not depend
on the frame's height (with all tables in shared memory four took 2.4 times one, without 1.3
times; 1.8 is between).
"""
import numpy as np
import pytest

import bdcudatag
import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CONFIG = dict(min_tag_pixels=4, min_cluster_pixels=4)
SIZES = [(64, 8192), (64, 8193), (48, 8200), (32, 16384), (640, 480), (32, 16)]


def boxes(width, height, step=20, size=10):
    img = np.full((height, width), 220, np.uint8)
    for k, y in enumerate(range(8, height - size - 2, step)):
        for x in range(8, width - size - 2, step):
            s = size - k % 5  # several area bins
            img[y:y + s, x:x + s] = 30
            img[y + 2:y + s - 2, x + 2:x + s - 2] = 220
    return img


def check(batch, frames):
    for i, f in enumerate(frames):
        ref = oracle.Frame(f, 0, oracle.default_config(**CONFIG))
        nc = ref.candidate_count
        assert batch.counts(i)[0] == ref.counts()[0]
        assert np.array_equal(batch.stage(i, "candidates")[:nc], ref.stage("candidates"))


@pytest.mark.parametrize("persistent", [0, 1])
@pytest.mark.parametrize("sizes", [SIZES] + [[s] for s in SIZES[:4]])
def test_candidates(sizes, persistent):
    frames = [boxes(w, h) for w, h in sizes]
    batch = bdcudatag.Batch([(w, h, 1) for w, h in sizes], bdcudatag.default_config(**CONFIG))
    batch.set_launch(persistent=persistent)
    batch.detect(frames)
    check(batch, frames)


def test_time():
    frame = torch.from_numpy(boxes(1280, 16384, 40, 20)).cuda()
    times = []
    for count in (1, 4):
        batch = bdcudatag.Batch([(1280, 16384, 1)] * count)
        times.append(min(batch.profile_device([frame] * count)["cand_count"] for _ in range(20)))
    assert times[1] <= 1.8 * times[0]
