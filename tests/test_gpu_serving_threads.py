"""A server that several threads submit to at once (gpu): two threads a camera, tight
rows, rows with a gap and page-locked frames in turn, the memory overwritten as soon as a
submit of a pageable frame returns.  Results bit for bit those of the oracle."""
import threading

import numpy as np
import pytest

import bdcudatag
import oracle
import scenes
from gpu_checks import same_records

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

SIZES = [(160, 120), (640, 480), (1283, 820), (1920, 1080)]  # below and above 1 MiB
ROUNDS = 6


@pytest.mark.parametrize("room", [False, True])
@pytest.mark.parametrize("pad", [0, 7])
def test_frames_in_device_memory(pad, room):
    """Copied at submit like pageable ones, whatever way those of the same shape take."""
    cameras = [(w, h, 1) for w, h in SIZES]
    plan = bdcudatag.Batch(cameras).device_bytes()
    server = bdcudatag.Server(cameras, device_budget=plan + (64 << 20 if room else 0), max_batches=1, queue_depth=12)
    tickets = []
    for c, (w, h) in enumerate(SIZES):
        frame = scenes.ref_scenes(w, h, 1)[0][0]
        rows = torch.full((h, w + pad), 255, dtype=torch.uint8, device="cuda")
        rows[:, :w] = torch.from_numpy(np.ascontiguousarray(frame)).cuda()
        torch.cuda.synchronize()
        tickets.append((server.submit(c, rows, w + pad), frame))
        assert tickets[-1][0] >= 0, bdcudatag.last_error()
        rows.zero_()
        torch.cuda.synchronize()
    for ticket, frame in tickets:
        rc, found, out, _ = server.wait(ticket)
        n, records = oracle.Frame(np.ascontiguousarray(frame), 0).detections()
        assert rc == 1 and found[0] == n
        same_records(out[0, :n], records)
    server.close()


@pytest.mark.parametrize("room", [False, True])  # request buffers in host memory, in device memory
def test_threads(room):
    cameras = [(w, h, 1) for w, h in SIZES]
    plan = bdcudatag.Batch(cameras).device_bytes()
    server = bdcudatag.Server(cameras, device_budget=plan + (64 << 20 if room else 0), max_batches=1, queue_depth=4)
    frames = [scenes.ref_scenes(w, h, 2)[0] for w, h in SIZES]
    want = [[oracle.Frame(np.ascontiguousarray(f), 0).detections() for f in camera] for camera in frames]
    errors = []
    barrier = threading.Barrier(2 * len(SIZES))

    def work(camera, which):
        try:
            w, h = SIZES[camera]
            n, records = want[camera][which]
            for k in range(ROUNDS):
                pad, pinned = (0, 7, 0)[k % 3], k % 3 == 2
                rows = torch.full((h, w + pad), 255, dtype=torch.uint8, pin_memory=pinned)
                rows[:, :w] = torch.from_numpy(np.ascontiguousarray(frames[camera][which]))
                barrier.wait()
                ticket = server.submit(camera, rows, w + pad)
                assert ticket >= 0, bdcudatag.last_error()
                if not pinned:
                    rows.zero_()
                rc, found, out, _ = server.wait(ticket)
                assert rc == 1 and found[0] == n
                same_records(out[0, :n], records)
        except Exception as e:  # noqa: BLE001 -- told by the main thread
            errors.append(repr(e))
            barrier.abort()

    threads = [threading.Thread(target=work, args=(c, k)) for c in range(len(SIZES)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert server.stats().completed == ROUNDS * len(threads)
    server.close()
