"""Pageable frames go to the device straight from the caller's memory, through
the staging buffer when their rows have a gap and they are small (gpu): both,
mixed with page-locked frames, on the plan's and on a caller's stream, and a
server with its request buffers in device and in host memory.  The memory is
overwritten as soon as the submit returns; results against the oracle."""
import numpy as np
import pytest

import bdcudatag
import oracle
import scenes
from gpu_checks import same_records

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SIZES = [(160, 120), (640, 480), (1280, 820)]  # below, below and above the bound of 1 MiB


def with_rows(frame, pad, pinned):
    h, w = frame.shape
    rows = torch.full((h, w + pad), 255, dtype=torch.uint8, pin_memory=pinned)
    rows[:, :w] = torch.from_numpy(np.ascontiguousarray(frame))
    return rows


def check(frame, found, out):
    for family in (0, 1):
        n, want = oracle.Frame(np.ascontiguousarray(frame), family).detections()
        assert found[family] == n
        same_records(out[family, :n], want)


@pytest.mark.parametrize("own_stream", [False, True])
@pytest.mark.parametrize("pad", [0, 7])
@pytest.mark.parametrize("pinned", [(0, 0, 0), (0, 1, 0), (1, 0, 1)])
def test_batch(pinned, pad, own_stream):
    frames = [scenes.ref_scenes(w, h, 2)[0] for w, h in SIZES]
    batch = bdcudatag.Batch([(w, h, 3) for w, h in SIZES])
    stream = torch.cuda.Stream() if own_stream else None
    batch.set_stream(stream)
    for call in range(2):
        rows = [with_rows(f[call], pad, bool(p)) for f, p in zip(frames, pinned)]
        batch.submit(rows, [w + pad for w, _ in SIZES])
        for r, p in zip(rows, pinned):
            if not p:
                r.zero_()
        found, out = batch.wait()
        for k, f in enumerate(frames):
            check(f[call], found[k], out[k])


@pytest.mark.parametrize("room", [False, True])
@pytest.mark.parametrize("pad", [0, 7])
def test_server(pad, room):
    cameras = [(w, h, 3) for w, h in SIZES]
    plan = bdcudatag.Batch(cameras).device_bytes()
    server = bdcudatag.Server(cameras, device_budget=plan + (64 << 20 if room else 0), max_batches=1,
                              queue_depth=2)
    frames = [scenes.ref_scenes(w, h, 2)[0] for w, h in SIZES]
    for _ in range(2):  # the request buffers are used again
        tickets = []
        for call in range(2):
            for c, f in enumerate(frames):
                rows = with_rows(f[call], pad, False)
                ticket = server.submit(c, rows, SIZES[c][0] + pad)
                assert ticket >= 0
                rows.zero_()
                tickets.append((ticket, f[call]))
        for ticket, frame in tickets:
            rc, found, out, _ = server.wait(ticket)
            assert rc == 1
            check(frame, found, out)
    server.close()
