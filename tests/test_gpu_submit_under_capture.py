"""Submits under a stream capture (gpu).  A plan with CUDA graphs refuses them, and works as
before afterwards.  A plan without takes them: the copies and launches become part
of the caller's graph, whose replays read pageable frames in the staging buffer, where the
submit left them; page-locked and device frames are read where they are.  Results of a replay are
there once the caller's stream is done (a first wait reports that the batch's event
was captured, a second one reads them).
"""
import numpy as np
import pytest

import bdcudatag
import oracle
import scenes
from gpu_checks import same_records

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

W, H = 640, 480


def frames(kind, images):
    rows = np.stack(images)
    if kind == "strided":
        rows = np.pad(rows, ((0, 0), (0, 0), (0, 7)))
    t = torch.from_numpy(np.ascontiguousarray(rows))
    return t.cuda() if kind == "device" else t.pin_memory() if kind == "pinned" else t


def check(found, out, image):
    n, want = oracle.Frame(np.ascontiguousarray(image), 0).detections()
    assert found[0, 0] == n
    same_records(out[0, 0, :n], want)


@pytest.mark.parametrize("kind", ["pageable", "strided", "pinned", "device"])
@pytest.mark.parametrize("graph", [0, 1])
def test_capture(kind, graph):
    images = scenes.ref_scenes(W, H, 2)[0]
    batch = bdcudatag.Batch([(W, H, 1)], bdcudatag.default_config(use_cuda_graph=graph))
    stream = torch.cuda.Stream()
    batch.set_stream(stream)
    source, stride, device = frames(kind, images), W + (7 if kind == "strided" else 0), kind == "device"
    captured = torch.cuda.CUDAGraph()
    refused = None
    try:
        with torch.cuda.graph(captured, stream=stream, capture_error_mode="relaxed"):
            try:
                batch.submit([source[0]], [stride], device=device)
            except RuntimeError as e:
                refused = e
    except Exception:  # noqa: BLE001 -- the refused submit ended the capture
        assert refused
    assert (refused is not None) == (graph == 1)
    if not graph:
        # The staged copy is the submit's; the others follow the caller's memory.
        source[0] = source[1].clone()
        torch.cuda.synchronize()
        shown = images[0] if kind in ("pageable", "strided") else images[1]
        for _ in range(2):
            captured.replay()
        torch.cuda.synchronize()
        with pytest.raises(RuntimeError):
            batch.wait()
        check(*batch.wait(), shown)
    if kind in ("pageable", "strided") or graph:
        check(*batch.detect([source[1]], [stride], device=device), images[1])
