"""Many candidates in one band cost a pass over its runs, not one over their pairs
(gpu): bands of 512 and fewer are ranked by comparing pairs in shared memory, larger
ones in slot order.  900 candidates of a band have twice the runs of 450; comparing
their pairs took six times as long, so four times is between.  The least of many runs.
Results at several sizes beyond 512 against the oracle.
"""
import numpy as np
import pytest

import bdcudatag
import oracle
from gpu_checks import check_frame

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CONFIG = dict(min_tag_pixels=4, min_cluster_pixels=4)


def boxes(width, height, step, size, every=1, rows=(9,)):
    """Hollow dark squares `step` pixels apart, every `every`-th a candidate and the others solid."""
    img = np.full((height, width), 220, np.uint8)
    for y in rows:
        for k, x in enumerate(range(8, width - size - 2, step)):
            img[y:y + size, x:x + size] = 30
            if k % every == 0:
                img[y + 2:y + size - 2, x + 2:x + size - 2] = 220
    return img


def stage_time(img):
    h, w = img.shape
    batch = bdcudatag.Batch([(w, h, 1)], bdcudatag.default_config(**CONFIG))
    frame = torch.from_numpy(img).cuda()
    times = [batch.profile_device([frame])["cand_count"] for _ in range(20)]
    return min(times), int(batch.counts(0)[0])


def test_time():
    few, n_few = stage_time(boxes(8192, 32, 9, 6, every=2))
    many, n_many = stage_time(boxes(8192, 32, 9, 6))
    assert n_few <= 512 < 2 * 400 < n_many
    assert many <= 4 * few


@pytest.mark.parametrize("width,step,size,rows", [
    (8192, 9, 6, (9,)),
    (8192, 15, 6, (9,)),            # 545
    (6000, 7, 5, (9, 17)),          # two such bands
    (8190, 10, 6, (9, 25)),
])
@pytest.mark.parametrize("threads", ["wide", "batch"])
def test_results(width, step, size, rows, threads):
    img = boxes(width, 40, step, size, rows=rows)
    if threads == "wide":  # 512 threads a band
        check_frame(img, 1, bdcudatag.default_config(**CONFIG), oracle.default_config(**CONFIG))
        return
    # Beside enough bands for 256 threads each, and by the persistent kernel.
    others = [(320, 2000, 1)] * 2
    batch = bdcudatag.Batch([(width, 40, 2)] + others, bdcudatag.default_config(**CONFIG))
    frames = [img] + [np.full((h, w), 128, np.uint8) for w, h, _ in others]
    ref = oracle.Frame(img, 1, oracle.default_config(**CONFIG))
    for persistent in (0, 1):
        batch.set_launch(persistent=persistent)
        batch.detect(frames)
        nc = ref.candidate_count
        assert np.array_equal(batch.stage(0, "candidates")[:nc], ref.stage("candidates"))
