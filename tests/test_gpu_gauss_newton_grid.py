"""One Gauss-Newton step over every shape of the sample grid (gpu): side lengths
below, at and above a warp's block of 8 columns and the 80 columns of ten warps, with given and with
measured levels, quads across the frame's edge and a degenerate one, against the
same step in 64 bits.

Tolerance: sums over the samples carry about 1e-6 of their size (FP32, a few
hundred to 65,536 terms in a tree), the damped normal equations of these textures
have condition numbers below 1e3, and a step is at most 2 px a coordinate: 2e-3 px.
The loss is a sum of squares: 1e-4 of itself.
"""
import numpy as np
import pytest

import bdcudatag

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

W, H = 320, 240


def step64(image, corners, template, samples, levels):
    """(corners after one damped step, loss before it) of one quad, numpy FP64."""
    cells = template.shape[0]
    i = np.arange(cells * samples)
    line = ((i // samples - 1) + (i % samples + 0.5) / samples) / (cells - 2)
    v, u = (a.ravel() for a in np.meshgrid(line, line, indexing="ij"))
    white = np.kron(template, np.ones((samples, samples))).ravel() != 0

    def homography(c):
        x0, y0, x1, y1, x2, y2, x3, y3 = c
        dx1, dx2, dx3 = x1 - x2, x3 - x2, x0 - x1 + x2 - x3
        dy1, dy2, dy3 = y1 - y2, y3 - y2, y0 - y1 + y2 - y3
        det = dx1 * dy2 - dx2 * dy1
        g, k = (dx3 * dy2 - dx2 * dy3) / det, (dx1 * dy3 - dx3 * dy1) / det
        return np.array([x1 - x0 + g * x1, x3 - x0 + k * x3, x0, y1 - y0 + g * y1, y3 - y0 + k * y3, y0, g, k])

    def values(c):
        h = homography(c)
        den = h[6] * u + h[7] * v + 1
        return (h[0] * u + h[1] * v + h[2]) / den, (h[3] * u + h[4] * v + h[5]) / den, den

    x, y, den = values(corners)
    inside = (den > 1e-6) & (x >= 0) & (y >= 0) & (x < W - 1) & (y < H - 1)
    ix, iy = np.where(inside, x, 0).astype(int), np.where(inside, y, 0).astype(int)
    fx, fy = np.where(inside, x - ix, 0), np.where(inside, y - iy, 0)
    a, b, c, d = (image[iy + j, ix + k].astype(float) for j in (0, 1) for k in (0, 1))
    value = (a * (1 - fx) + b * fx) * (1 - fy) + (c * (1 - fx) + d * fx) * fy
    gx, gy = (b - a) * (1 - fy) + (d - c) * fy, (c - a) * (1 - fx) + (d - b) * fx
    jac = np.zeros((len(u), 8))
    for k in range(8):  # positions are smooth: central differences give their derivatives
        e = np.zeros(8)
        e[k] = 1e-4
        xp, yp, _ = values(corners + e)
        xm, ym, _ = values(corners - e)
        jac[:, k] = np.where(inside, gx * (xp - xm) / 2e-4 + gy * (yp - ym) / 2e-4, 0)
    if levels is None:
        levels = [value[inside & (white == w)].mean() for w in (False, True)]
    r = np.where(inside, value - np.where(white, levels[1], levels[0]), 0)
    m = jac.T @ jac
    m += 1e-4 * np.diag(np.diag(m))
    step = np.linalg.solve(m, -jac.T @ r)
    return corners + np.clip(step, -2, 2), 0.5 * (r * r).sum()


@pytest.mark.parametrize("measured", [True, False])
@pytest.mark.parametrize("cells,samples", [(4, 3), (8, 2), (5, 5), (8, 8), (10, 8), (11, 8), (16, 5), (16, 16)])
def test_one_step(cells, samples, measured):
    rng = np.random.default_rng(100 * cells + samples)
    noise = np.kron(rng.uniform(0, 255, (H // 8 + 2, W // 8 + 2)), np.ones((8, 8)))
    smooth = sum(noise[j:j + H, i:i + W] for j in range(8) for i in range(8)) / 64
    image = np.ascontiguousarray(smooth.astype(np.uint8))
    base = np.array([[60.3, 50.2], [200.7, 61.1], [190.4, 180.9], [70.8, 170.5]])
    quads = np.stack([base, base[::-1] * 0.9 + 7, base + [150.0, 90.0], np.array([[9.0, 9], [50, 50], [90, 90], [130, 130]])])
    quads = quads.reshape(4, 8).astype(np.float32)
    templates = rng.integers(0, 2, (4, cells, cells)).astype(np.uint8)
    templates[:, 0, 0], templates[:, 1, 1] = 0, 1  # both colours
    levels = None if measured else np.tile(np.array([[40.0, 200.0]], np.float32), (4, 1))
    im, te = torch.from_numpy(image[None]).cuda(), torch.from_numpy(templates).cuda()
    ix = torch.zeros(4, dtype=torch.int32, device="cuda")
    lv = None if measured else torch.from_numpy(levels).cuda()
    for iterations in (0, 1):
        co = torch.from_numpy(quads.copy()).cuda()
        loss = torch.full((4,), -1.0, device="cuda")
        args = bdcudatag.refine_args(im, co, te, ix, lv, samples)
        assert bdcudatag.lib().bd_refine_gauss_newton(args, co.data_ptr(), iterations, loss.data_ptr(), None) == 0
        got, got_loss = co.cpu().numpy(), loss.cpu().numpy()
        assert np.array_equal(got[3], quads[3]) and got_loss[3] == 0.0  # no homography: left as it is
        for k in range(3):
            want, before = step64(image, quads[k].astype(float), templates[k], samples,
                                  None if measured else levels[k])
            if iterations == 0:
                assert np.array_equal(got[k], quads[k])
                assert abs(got_loss[k] - before) <= 1e-4 * before
            else:
                assert np.abs(got[k] - want).max() <= 2e-3
