"""The work that programs have this library do, as cases that can be timed.

Every case goes through the public entry points (the C ABI and its ctypes
binding, bdcudatag.py).  The seed picks frames out of pools that the package's own
scene generator renders, with the benchmark's tag, noise and clutter distributions
(MIXED_1280 at 1280x800 is the benchmark's own pool of 600).  Frames of other sizes
are scenes of the reference's benchmark generator.  Frame sizes and batch
shapes are those of bench.py and of the tests, or generic odd ones.

kind            what a pass is
frame           one bd_detector call on one frame (the drop-in API)
rig             one bd_batch call on a fixed set of cameras
rig_stream      bd_batch_pipeline: one batch on each of `plans` batches, all in
                flight together, then the results of each
serve           one frame of every camera through a bd_server, then its results
refine_grad     photometric residuals and loss, then the adjoint (dL/dcorners
                and dL/dimages)
refine_gn       Gauss-Newton corner refinement
tile_stats      bd_tile_stats_device_noalloc on one frame
"""
import ctypes
import os
import sys
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

# Many batches run at once on streams of their own; as bench.py sets it.
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")
sys.path.insert(0, os.path.join(os.getcwd(), "bd-cudatag_gb300"))

import bdcudatag  # noqa: E402
import scenes  # noqa: E402

REF_SCENES = 0  # scene: the reference's benchmark set, at any size

# Frames in the pool of each scene set.
POOL = {scenes.EIGHT_TAGS_640: 600, scenes.MIXED_1280: 600, scenes.MULTI_SIZE: 600, scenes.SERVING: 300}
# Frames that no pass takes: each has a quad whose sampled contrast lies, by rounding alone, above the
# decoder's limit in one rotation and below it in another.  Earlier builds of the decoder do not
# return from such a quad.
LEFT_OUT = {
    (scenes.EIGHT_TAGS_640, 640, 480): {478},
    (scenes.MULTI_SIZE, 1283, 717): {233, 347},
    (scenes.MULTI_SIZE, 1280, 800): {435},
    (scenes.MULTI_SIZE, 1600, 1304): {45, 188, 320, 475, 518},
    (scenes.MULTI_SIZE, 1920, 1080): {66, 382, 420, 514},
    (scenes.SERVING, 1280, 800): {120},
    (scenes.SERVING, 1600, 1304): {13, 229, 247},
    (scenes.SERVING, 1920, 1080): {0, 22, 46, 53, 147, 195},
    (scenes.SERVING, 2560, 1440): {107, 132, 180, 193, 209, 229, 232},
    (scenes.SERVING, 3840, 2160): {22, 24, 46, 70, 99, 155, 170, 186, 195, 223, 232, 252, 291},
}

MIXED_SIZES = [(640, 480), (1280, 800), (1600, 1304), (1920, 1080)]
SERVE_SIZES = [(640, 480), (1280, 720), (1280, 800), (1600, 1304), (1920, 1080), (2560, 1440),
               (3840, 2160)]
FIELDS = ("id", "hamming", "decision_margin", "corners", "homography")
GN_ITERATIONS = 5
QUADS_PER_FRAME = {0: 6, 1: 2}  # tags of each family that a frame holds


def listed():
    return [
        # A program of the reference's C ABI: one 36h11 detector, pageable
        # 640x480 frames (the plain single-frame workload).
        dict(name="frame_640_host", kind="frame", width=640, height=480, family=0, source="host", pad=0,
             scene=scenes.EIGHT_TAGS_640, refine_edges=True),
        # The smallest calls: a thumbnail already on the device, where
        # latency and launches are all there is.
        dict(name="frame_small_device", kind="frame", width=192, height=144, family=1, source="device",
             pad=0, scene=scenes.MULTI_SIZE, refine_edges=True),
        # A cropped view of a larger image: odd size, rows that start at no
        # aligned address.
        dict(name="frame_odd_device", kind="frame", width=1283, height=717, family=0, source="device",
             pad=10, scene=scenes.MULTI_SIZE, refine_edges=True),
        # The largest camera of the serving mix, from pageable host memory.
        dict(name="frame_4k_host", kind="frame", width=3840, height=2160, family=0, source="host", pad=0,
             scene=scenes.SERVING, refine_edges=True),
        # A four-camera rig, one synchronous batch at a time (a control loop
        # that needs the answer before it goes on).
        dict(name="rig4_1280_device", kind="rig", sizes="1280x800x4", families=3, source="device",
             scene=scenes.MIXED_1280),
        # The headline workload: such batches with many in flight, frames
        # resident on the device ...
        dict(name="rig4_1280_stream_device", kind="rig_stream", plans=16, sizes="1280x800x4", families=3,
             source="device", scene=scenes.MIXED_1280),
        # ... and copied from page-locked host memory in every pass.
        dict(name="rig4_1280_stream_pinned", kind="rig_stream", plans=16, sizes="1280x800x4", families=3,
             source="pinned", scene=scenes.MIXED_1280),
        # 16 cameras of four sizes in one batch.
        dict(name="rig16_mixed_device", kind="rig", sizes="mixed x4", families=3, source="device",
             scene=scenes.MULTI_SIZE),
        # A server of six cameras from 640x480 to 3840x2160, a frame of each.
        dict(name="serve_6_cameras", kind="serve", cameras=6, first=0, scene=scenes.SERVING),
        # One step of a program that differentiates through the photometric
        # residual of 256 detected quads.
        dict(name="refine_grad_256", kind="refine_grad", quads=256, family=0, samples=8),
        # Corner refinement of 256 detected quads.
        dict(name="refine_gn_256", kind="refine_gn", quads=256, family=0, samples=8),
        # First-stage statistics for a caller that may not allocate.
        dict(name="tile_stats_1080p", kind="tile_stats", width=1920, height=1080, pad=0,
             scene=scenes.MULTI_SIZE),
    ]


def _size(rng, lo, hi):
    """A width spread over its logarithm, odd ones among them, and a height
    of an ordinary aspect."""
    w = int(round(lo * (hi / lo) ** rng.random()))
    h = max(32, int(w * rng.uniform(0.5, 0.85)))
    return w, h


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "rig", "rig", "rig_stream", "serve", "refine_grad",
                       "refine_gn", "tile_stats"])
    if kind == "frame":
        w, h = _size(rng, 64, 2800)
        return dict(kind=kind, width=w, height=h, family=rng.randrange(2),
                    source=rng.choice(["host", "device", "pinned"]), pad=rng.choice([0, 0, 6, 32]),
                    scene=REF_SCENES, refine_edges=rng.random() < 0.85)
    if kind in ("rig", "rig_stream"):
        w, h = _size(rng, 320, 1600)
        n = rng.randint(1, 8)
        case = dict(kind=kind, sizes="%dx%dx%d" % (w, h, n), families=rng.randint(1, 3),
                    source=rng.choice(["device", "pinned"]), scene=REF_SCENES)
        if kind == "rig_stream":
            case["plans"] = rng.randint(2, max(2, min(16, int(40e6 / (w * h * n)))))
        return case
    if kind == "serve":
        n = rng.randint(1, 5)
        return dict(kind=kind, cameras=n, first=rng.randrange(7 - n) if n < 3 else 0, scene=scenes.SERVING)
    if kind == "tile_stats":
        w, h = _size(rng, 64, 4096)
        return dict(kind=kind, width=w, height=h, pad=rng.choice([0, 0, 6, 32]), scene=REF_SCENES)
    family = rng.randrange(2)
    return dict(kind=kind, quads=int(round(4 * (64 if family == 0 else 16) ** rng.random())), family=family,
                samples=rng.choice([3, 4, 6, 8, 8]))


# --- inputs ------------------------------------------------------------------


def _sizes(case):
    if case["kind"] == "serve":
        return SERVE_SIZES[case["first"]:case["first"] + case["cameras"]]
    if case["sizes"].startswith("mixed x"):
        return MIXED_SIZES * int(case["sizes"][len("mixed x"):])
    w, h, n = (int(v) for v in case["sizes"].split("x"))
    return [(w, h)] * n


def _render(case, seed, sizes):
    """One frame for each size: another one of the pool for each frame of a size."""
    scene = case["scene"]
    if scene == REF_SCENES:
        (w, h), = set(sizes)
        return list(scenes.ref_scenes(w, h, len(sizes), seed & 0xffffffff)[0])
    rng = np.random.default_rng(seed)
    order = {}
    for size in sorted(set(sizes)):
        left_out = LEFT_OUT.get((scene,) + size, ())
        order[size] = [i for i in rng.permutation(POOL[scene]).tolist() if i not in left_out]
    todo = [(order[size].pop(), size) for size in sizes]
    with ThreadPoolExecutor(os.cpu_count() or 8) as pool:
        return list(pool.map(lambda t: scenes.render_scene(scene, t[0], *t[1])[0], todo))


def _with_stride(frame, pad):
    """The frame as the left part of rows that are `pad` bytes longer."""
    if not pad:
        return np.ascontiguousarray(frame)
    h, w = frame.shape
    rows = np.zeros((h, w + pad), dtype=np.uint8)
    rows[:, :w] = frame
    return rows


def _place(frame, source):
    if source == "host":
        return frame
    t = torch.from_numpy(np.ascontiguousarray(frame))
    return t.pin_memory() if source == "pinned" else t.cuda()


def _quads(case, seed):
    """Quads as a detector hands them on: ground-truth corners moved by up to
    1.5 px, with the frames that they lie in."""
    frames_wanted = -(-case["quads"] // QUADS_PER_FRAME[case["family"]])
    images, index, corners, templates = [], [], [], []
    rng = np.random.default_rng(seed)
    base = 1_000_000 + 4096 * seed
    while len(corners) < case["quads"]:
        got, truth = scenes.render_many(scenes.REFINE_1280, [(1280, 800)] * frames_wanted,
                                        threads=os.cpu_count() or 8, base=base)
        base += frames_wanted
        for frame, tags in zip(got, truth):
            mine = [t for t in tags if t.family == case["family"]]
            if not mine or len(corners) >= case["quads"]:
                continue
            for t in mine:
                corners.append(t.corners.reshape(8))
                templates.append(bdcudatag.tag_template(t.family, t.id))
                index.append(len(images))
            images.append(frame)
    n = case["quads"]
    corners = np.stack(corners[:n])
    corners = (corners + rng.uniform(-1.5, 1.5, corners.shape)).astype(np.float32)
    levels = np.tile(np.array([[30.0, 220.0]], np.float32), (n, 1))
    return dict(images=torch.from_numpy(np.stack(images)).cuda(), corners=torch.from_numpy(corners).cuda(),
                templates=torch.from_numpy(np.stack(templates[:n])).cuda(),
                index=torch.from_numpy(np.array(index[:n], np.int32)).cuda(),
                levels=torch.from_numpy(levels).cuda())


def prepare(case, seed):
    kind = case["kind"]
    state = dict(kind=kind)
    if kind == "frame":
        w, h = case["width"], case["height"]
        frame = _with_stride(_render(case, seed, [(w, h)])[0], case["pad"])
        config = bdcudatag.default_config(refine_edges=1 if case["refine_edges"] else 0)
        state.update(detector=bdcudatag.Detector(case["family"], w, h, config),
                     frame=_place(frame, case["source"]), stride=w + case["pad"],
                     device=case["source"] == "device")
    elif kind == "rig":
        sizes = _sizes(case)
        state.update(batch=bdcudatag.Batch([(w, h, case["families"]) for w, h in sizes]),
                     frames=[_place(f, case["source"]) for f in _render(case, seed, sizes)],
                     strides=[w for w, _ in sizes], device=case["source"] == "device")
    elif kind == "rig_stream":
        sizes = _sizes(case)
        n, plans = len(sizes), case["plans"]
        frames = [_place(f, case["source"]) for f in _render(case, seed, sizes * plans)]
        batches = [bdcudatag.Batch([(w, h, case["families"]) for w, h in sizes]) for _ in range(plans)]
        state.update(batches=batches, sets=[frames[k * n:(k + 1) * n] for k in range(plans)],
                     strides=[w for w, _ in sizes], device=case["source"] == "device",
                     found=np.zeros((plans, n, 2), np.int32),
                     records=np.zeros((plans, n, 2, batches[0].max_detections),
                                      bdcudatag.DETECTION_DTYPE))
    elif kind == "serve":
        sizes = _sizes(case)
        state.update(server=bdcudatag.Server([(w, h, 3) for w, h in sizes]),
                     frames=_render(case, seed, sizes))
    elif kind == "tile_stats":
        w, h = case["width"], case["height"]
        tiles = (-(-h // 8), -(-w // 8))
        state.update(frame=_place(_with_stride(_render(case, seed, [(w, h)])[0], case["pad"]), "device"),
                     width=w, height=h, stride=w + case["pad"],
                     tile_min=torch.zeros(tiles, dtype=torch.uint8, device="cuda"),
                     tile_max=torch.zeros(tiles, dtype=torch.uint8, device="cuda"),
                     refs=torch.zeros(3, dtype=torch.int32, device="cuda"))
    else:
        state.update(_quads(case, seed), samples=case["samples"])
        n, cells = case["quads"], 10 if case["family"] == 0 else 8
        if kind == "refine_grad":
            state.update(residuals=torch.empty((n, (cells * case["samples"]) ** 2), device="cuda"),
                         loss=torch.empty(n, device="cuda"), grad_corners=torch.empty((n, 8), device="cuda"),
                         grad_images=torch.empty(state["images"].shape, device="cuda"))
        else:
            state.update(refined=torch.empty((n, 8), device="cuda"), loss=torch.empty(n, device="cuda"))
    torch.cuda.synchronize()
    return state


# --- one pass ----------------------------------------------------------------


def _fields(found, records):
    return [found] + [records[f] for f in FIELDS]


def _ok(rc):
    if rc != 0:
        raise RuntimeError("%d: %s" % (rc, bdcudatag.last_error()))


def run(state):
    kind = state["kind"]
    if kind == "frame":
        detector = state["detector"]
        detect = detector.detect_device if state["device"] else detector.detect
        found, _ = detect(state["frame"], state["stride"])
        s = detector.stats()
        return _fields(found, detector.out) + [s.runs, s.candidates, s.quads, s.roi_rows]
    if kind == "rig":
        return _fields(*state["batch"].detect(state["frames"], state["strides"], device=state["device"]))
    if kind == "rig_stream":
        batches, found, records = state["batches"], state["found"], state["records"]
        bdcudatag.pipeline(batches, state["sets"], state["strides"], len(batches), state["device"])
        for k, batch in enumerate(batches):
            _ok(bdcudatag.lib().bd_batch_wait(batch.handle, records[k].ctypes.data, found[k].ctypes.data))
        return _fields(found, records)
    if kind == "serve":
        server, out = state["server"], []
        tickets = [server.submit(c, f) for c, f in enumerate(state["frames"])]
        for ticket in tickets:
            status, found, records, _ = server.wait(ticket)
            out.append([status] + _fields(found, records))
        return out
    if kind == "tile_stats":
        _ok(bdcudatag.lib().bd_tile_stats_device_noalloc(
            state["frame"].data_ptr(), state["width"], state["height"], state["stride"],
            state["tile_min"].data_ptr(), state["tile_max"].data_ptr(), state["refs"].data_ptr(),
            torch.cuda.current_stream().cuda_stream))
        return [state["tile_min"], state["tile_max"], state["refs"]]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "refine_grad":
        args = bdcudatag.refine_args(state["images"], state["corners"], state["templates"], state["index"],
                                     state["levels"], state["samples"])
        res, loss = state["residuals"], state["loss"]
        gc, gi = state["grad_corners"], state["grad_images"]
        _ok(bdcudatag.lib().bd_refine_forward(args, res.data_ptr(), loss.data_ptr(), stream))
        gi.zero_()  # the adjoint adds to it
        _ok(bdcudatag.lib().bd_refine_backward(args, res.data_ptr(), gc.data_ptr(), gi.data_ptr(), stream))
        return [res, loss, gc, gi]
    corners = state["refined"].copy_(state["corners"])
    args = bdcudatag.refine_args(state["images"], corners, state["templates"], state["index"], None,
                                 state["samples"])
    _ok(bdcudatag.lib().bd_refine_gauss_newton(args, corners.data_ptr(), GN_ITERATIONS,
                                               state["loss"].data_ptr(), stream))
    return [corners, state["loss"]]


# --- what a pass cannot do without --------------------------------------------


def work(case):
    kind = case["kind"]
    record = ctypes.sizeof(bdcudatag.Detection)
    if kind == "frame":
        return {"bytes": case["width"] * case["height"] + 8 * record, "flops": 0}
    if kind in ("rig", "rig_stream", "serve"):
        sizes = _sizes(case) * case.get("plans", 1)
        return {"bytes": sum(w * h + 8 * record for w, h in sizes), "flops": 0}
    if kind == "tile_stats":
        return {"bytes": case["width"] * case["height"] * (1 + 2 / 64), "flops": 0}
    n, cells = case["quads"], 10 if case["family"] == 0 else 8
    samples = n * (cells * case["samples"]) ** 2
    if kind == "refine_grad":
        # Residuals written and read, gradients of the frames written, the
        # frames' tags read (at least one byte per sample's cell side); 35
        # operations a residual, 120 its adjoint.
        frames = -(-n // QUADS_PER_FRAME[case["family"]]) * 1280 * 800
        return {"bytes": 8 * samples + 4 * frames, "flops": 155 * samples}
    # Per iteration and sample: the residual with its 8 derivatives (155), 36 + 8
    # products of the normal equations (88), and the photometric levels.
    return {"bytes": samples + n * (cells * cells + 72), "flops": 250 * samples * (GN_ITERATIONS + 1)}


# --- the same in 64 bits -------------------------------------------------------


def _homography(c):
    x0, y0, x1, y1, x2, y2, x3, y3 = c.unbind(-1)
    dx1, dx2, dx3 = x1 - x2, x3 - x2, x0 - x1 + x2 - x3
    dy1, dy2, dy3 = y1 - y2, y3 - y2, y0 - y1 + y2 - y3
    det = dx1 * dy2 - dx2 * dy1
    g = (dx3 * dy2 - dx2 * dy3) / det
    k = (dx1 * dy3 - dx3 * dy1) / det
    return torch.stack([x1 - x0 + g * x1, x3 - x0 + k * x3, x0, y1 - y0 + g * y1, y3 - y0 + k * y3, y0, g, k],
                       dim=-1)


def _grid(cells, samples, device):
    s = torch.arange(cells * cells * samples * samples, device=device)
    cell, sub = s // (samples * samples), s % (samples * samples)
    u = ((cell % cells - 1).double() + ((sub % samples).double() + 0.5) / samples) / (cells - 2)
    v = ((cell // cells - 1).double() + ((sub // samples).double() + 0.5) / samples) / (cells - 2)
    return cell, u, v


def _sampled(q, corners):
    """(inside, frame value, white cell, d value / d corners, where it lies) of every sample, in 64 bits."""
    flat = q["images"].reshape(-1)
    _, height, width = q["images"].shape
    cell, u, v = _grid(q["templates"].shape[-1], q["samples"], corners.device)
    h = _homography(corners)[:, :, None]
    den = h[:, 6] * u + h[:, 7] * v + 1.0
    x = (h[:, 0] * u + h[:, 1] * v + h[:, 2]) / den
    y = (h[:, 3] * u + h[:, 4] * v + h[:, 5]) / den
    inside = (den > 1e-6) & (x >= 0) & (y >= 0) & (x < width - 1) & (y < height - 1)
    xc, yc = torch.where(inside, x, torch.zeros_like(x)), torch.where(inside, y, torch.zeros_like(y))
    ix, iy = xc.floor().long(), yc.floor().long()
    fx, fy = xc - ix, yc - iy
    at = q["index"].long()[:, None] * (height * width) + iy * width + ix
    a, b, c, d = (flat[at + o].double() for o in (0, 1, width, width + 1))
    value = (a * (1 - fx) + b * fx) * (1 - fy) + (c * (1 - fx) + d * fx) * fy
    white = q["templates"].reshape(corners.shape[0], -1)[:, cell] != 0
    gx = (b - a) * (1 - fy) + (d - c) * fy
    gy = (c * (1 - fx) + d * fx) - (a * (1 - fx) + b * fx)
    dh = torch.func.vmap(torch.func.jacfwd(_homography))(corners)  # n, 8 of h, 8 of c
    jac = []
    for k in range(8):
        e = dh[:, :, k, None]
        dden = e[:, 6] * u + e[:, 7] * v
        dx = (e[:, 0] * u + e[:, 1] * v + e[:, 2] - x * dden) / den
        dy = (e[:, 3] * u + e[:, 4] * v + e[:, 5] - y * dden) / den
        jac.append(torch.where(inside, gx * dx + gy * dy, torch.zeros_like(x)))
    return inside, value, white, torch.stack(jac, -1), (at, width, fx, fy)


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("refine_grad", "refine_gn"):
        return None  # whole numbers, or values of discrete decisions
    q = dict(_quads(case, seed), samples=case["samples"])
    corners = q["corners"].double()
    zero = torch.zeros((), dtype=torch.float64, device=corners.device)
    if kind == "refine_grad":
        inside, value, white, jac, (at, width, fx, fy) = _sampled(q, corners)
        lo, hi = q["levels"].double().unbind(1)
        r = torch.where(inside, value - torch.where(white, hi[:, None], lo[:, None]), zero)
        gi = torch.zeros(q["images"].numel(), dtype=torch.float64, device=corners.device)
        for o, w in ((0, (1 - fx) * (1 - fy)), (1, fx * (1 - fy)), (width, (1 - fx) * fy),
                     (width + 1, fx * fy)):
            gi.index_add_(0, (at + o).reshape(-1), (r * w).reshape(-1))
        return [r, 0.5 * (r * r).sum(1), (r[:, :, None] * jac).sum(1), gi.reshape(q["images"].shape)]
    for iteration in range(GN_ITERATIONS + 1):
        inside, value, white, jac, _ = _sampled(q, corners)
        lo, hi = (torch.where(m, value, zero).sum(1) / m.sum(1) for m in (inside & ~white, inside & white))
        r = torch.where(inside, value - torch.where(white, hi[:, None], lo[:, None]), zero)
        loss = 0.5 * (r * r).sum(1)
        if iteration < GN_ITERATIONS:
            jtj = jac.transpose(1, 2) @ jac
            jtr = (jac * r[:, :, None]).sum(1)
            damped = jtj + 1e-4 * torch.diag_embed(torch.diagonal(jtj, dim1=1, dim2=2))
            step = torch.cholesky_solve(-jtr[:, :, None], torch.linalg.cholesky(damped))[:, :, 0]
            corners = corners + step.clamp(-2.0, 2.0)
    return [corners, loss]
