"""Region sums of bands with few and many roots, around the bound from which a
band adds them up in shared memory first, and with more components than that
table holds (gpu), against the oracle."""
import numpy as np
import pytest

import bdcudatag
import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("lines,joined", [(100, 1), (511, 1), (512, 1), (513, 1), (513, 16), (1500, 1), (1500, 513)])
def test_lines(lines, joined):
    """Vertical lines from top to bottom, one component each, `joined` of them at a
    time by a bar across the frame's middle."""
    w, h = 2 * lines + 30, 60
    img = np.full((h, w), 220, np.uint8)
    img[4:h - 4, 10:10 + 2 * lines:2] = 30
    for first in range(0, lines, joined):
        last = min(first + joined, lines) - 1
        img[29:31, 10 + 2 * first:11 + 2 * last] = 30
    batch = bdcudatag.Batch([(w, h, 1)])
    batch.detect([torch.from_numpy(img).cuda()], [w], device=True)
    ref = oracle.Frame(img, 0)
    rc = batch.stage(0, "row_count")
    assert np.array_equal(rc, ref.stage("row_count"))
    valid = (np.arange(ref.row_cap)[None, :] < rc[:, None]).ravel()
    lab = batch.stage(0, "label")[valid]
    assert np.array_equal(lab, ref.stage("label")[valid])
    roots = np.unique(lab)
    assert len(roots) == -(-lines // joined)
    assert np.array_equal(batch.stage(0, "area")[roots], ref.stage("area")[roots])
    assert np.array_equal(batch.stage(0, "bbox").reshape(-1, 4)[roots], ref.stage("bbox").reshape(-1, 4)[roots])
