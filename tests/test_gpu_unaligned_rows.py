"""Rows at any address and frames of any width are binarized from whole words where
these lie inside the frame (gpu): offsets, gaps between rows and widths around the
words, the bits, runs and results against the oracle."""
import numpy as np
import pytest

import bdcudatag
import oracle
import scenes
from gpu_checks import same_records

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("offset", [0, 1, 3, 16])
@pytest.mark.parametrize("w,h,pad", [
    (16, 16, 0), (16, 17, 1), (31, 40, 0), (32, 40, 3), (33, 24, 16), (61, 33, 2), (64, 32, 0), (95, 41, 33),
    (157, 120, 0), (157, 120, 3), (160, 121, 16), (1283, 93, 10), (1311, 64, 1),
])
def test_rows(w, h, pad, offset):
    if w >= 157 and h >= 120:
        img = scenes.ref_scenes(w, h, 1)[0][0]
    else:
        rng = np.random.default_rng(w * h)
        img = np.kron(rng.integers(0, 256, ((h + 3) // 4, (w + 3) // 4)), np.ones((4, 4)))[:h, :w]
    img = np.ascontiguousarray(img.astype(np.uint8))
    stride = w + pad
    size = offset + (h - 1) * stride + w  # the frame ends where the buffer does
    flat = torch.full((size,), 255, dtype=torch.uint8)
    view = torch.as_strided(flat, (h, w), (stride, 1), offset)
    view[:] = torch.from_numpy(img)
    dev = flat.cuda()
    batch = bdcudatag.Batch([(w, h, 3)])
    found, out = batch.detect([dev.data_ptr() + offset], [stride], device=True)
    ref = oracle.Frame(img, 0)
    assert np.array_equal(batch.stage(0, "bits"), ref.stage("bits"))
    rc = batch.stage(0, "row_count")
    assert np.array_equal(rc, ref.stage("row_count"))
    valid = (np.arange(ref.row_cap)[None, :] < rc[:, None]).ravel()
    assert np.array_equal(batch.stage(0, "runs")[valid], ref.stage("runs")[valid])
    for family in (0, 1):
        n, want = oracle.Frame(img, family).detections()
        assert found[0, family] == n
        same_records(out[0, family, :n], want)
