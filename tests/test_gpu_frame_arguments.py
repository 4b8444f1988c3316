"""The frames of a call reach the kernels as an argument of the first one, which
is replaced in the captured graph for each call, and the records come back in
host memory (gpu): other frames, strides and frame counts from call to call,
with and without a graph, against the oracle."""
import numpy as np
import pytest

import bdcudatag
import oracle
import scenes
from gpu_checks import same_records

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("cameras", [1, 3, 64])
def test_frames_change_from_call_to_call(cameras, graph):
    w, h = 160, 120
    frames = scenes.ref_scenes(w, h, cameras + 2)[0]
    batch = bdcudatag.Batch([(w, h, 3)] * cameras, bdcudatag.default_config(use_cuda_graph=graph))
    other = bdcudatag.Batch([(w, h, 1)] * cameras)
    for call, pad in enumerate((0, 6, 0)):
        mine = []
        for k in range(cameras):
            rows = torch.zeros((h, w + pad), dtype=torch.uint8, device="cuda")
            rows[:, :w] = torch.from_numpy(frames[(k + call) % len(frames)])
            mine.append(rows)
        other.submit([torch.from_numpy(f).cuda() for f in frames[:cameras]], device=True)
        found, out = batch.detect(mine, [w + pad] * cameras, device=True)
        other.wait()
        for k in range(cameras):
            for family in (0, 1):
                n, want = oracle.Frame(np.ascontiguousarray(frames[(k + call) % len(frames)]), family).detections()
                assert found[k, family] == n
                same_records(out[k, family, :n], want)
