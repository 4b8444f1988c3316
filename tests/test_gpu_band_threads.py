"""Bands labelled, merged and summed by as many threads as their number and their
frames' width ask for (gpu): widths around the bounds of the rule, few and many bands,
bands that fit, that are cut into segments and that fall back, against the oracle."""
import numpy as np
import pytest

import bdcudatag
import oracle
from gpu_checks import same_records

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def patterns(w, h):
    rng = np.random.default_rng(w + h)
    out = [np.where(rng.random((h, w)) < p, 30, 220).astype(np.uint8) for p in (0.4, 0.6)]
    comb = np.full((h, w), 220, np.uint8)
    comb[4:h - 3, 5:w - 5:3] = 30
    comb[4:7, 5:w - 5] = 30
    return out + [comb]


@pytest.mark.parametrize("w,h,count", [(3072, 45, 3), (3073, 45, 3), (3840, 120, 3), (3105, 45, 64)])
def test_wide_bands(w, h, count):
    test_bands(w, h, count, 1024)


@pytest.mark.parametrize("band_cap", [256, 2048])
@pytest.mark.parametrize("w,h,count", [
    (1024, 45, 3), (1025, 45, 3), (1057, 45, 3), (2050, 45, 3),      # few bands
    (640, 45, 64), (1057, 45, 64), (2048, 45, 64), (2050, 45, 64),   # more than two per SM
])
def test_bands(w, h, count, band_cap):
    frames = patterns(w, h)
    batch = bdcudatag.Batch([(w, h, 1)] * count)
    batch.set_launch(band_cap=band_cap)
    dev = [torch.from_numpy(f).cuda() for f in frames]
    found, out = batch.detect([dev[i % 3] for i in range(count)], [w] * count, device=True)
    for i in list(range(3)) + [count - 1]:
        ref = oracle.Frame(frames[i % 3], 0)
        rc = batch.stage(i, "row_count")
        assert np.array_equal(rc, ref.stage("row_count"))
        valid = (np.arange(ref.row_cap)[None, :] < rc[:, None]).ravel()
        assert np.array_equal(batch.stage(i, "runs")[valid], ref.stage("runs")[valid])
        lab = batch.stage(i, "label")[valid]
        assert np.array_equal(lab, ref.stage("label")[valid])
        roots = np.unique(lab)
        assert np.array_equal(batch.stage(i, "area")[roots], ref.stage("area")[roots])
        assert np.array_equal(batch.stage(i, "bbox").reshape(-1, 4)[roots],
                              ref.stage("bbox").reshape(-1, 4)[roots])
        wn, want = ref.detections()
        assert found[i, 0] == wn
        same_records(out[i, 0, :wn], want)
