"""Loss of the Gauss-Newton refinement with measured levels where the residuals
are small beside the levels (gpu): frames of low contrast, cells of one value, and
steps after which the levels have moved by more than the residuals, against 64 bits.

Tolerances: positions are within 1e-5 px and values within 1.5e-5, so a residual
is within e = 1e-5 of the local gradient plus 1.5e-5, sample by sample and of either
sign.  Low contrast: 2e-5 / 0.3 over sqrt(1,024) samples, times two, is 4e-6 of the
loss; 2e-5.  Cells of one value: |r| <= 1e-4, so at most 5e-9 a sample.  Moved
levels: gradients of 82 a pixel, e = 8.4e-4, all of one sign, and so at most
e sum |r| + n e^2 / 2 <= e sqrt(2 n loss) + n e^2 / 2.
"""
import numpy as np
import pytest

import bdcudatag

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

W, H = 320, 240


def loss64(image, corners, template, samples):
    """Loss at the corners with the mean of each colour as its level, numpy FP64; all samples inside."""
    cells = template.shape[0]
    i = np.arange(cells * samples)
    line = ((i // samples - 1) + (i % samples + 0.5) / samples) / (cells - 2)
    v, u = (a.ravel() for a in np.meshgrid(line, line, indexing="ij"))
    white = np.kron(template, np.ones((samples, samples))).ravel() != 0
    x0, y0, x1, y1, x2, y2, x3, y3 = corners
    dx1, dx2, dx3 = x1 - x2, x3 - x2, x0 - x1 + x2 - x3
    dy1, dy2, dy3 = y1 - y2, y3 - y2, y0 - y1 + y2 - y3
    det = dx1 * dy2 - dx2 * dy1
    g, k = (dx3 * dy2 - dx2 * dy3) / det, (dx1 * dy3 - dx3 * dy1) / det
    den = g * u + k * v + 1
    x = ((x1 - x0 + g * x1) * u + (x3 - x0 + k * x3) * v + x0) / den
    y = ((y1 - y0 + g * y1) * u + (y3 - y0 + k * y3) * v + y0) / den
    assert x.min() >= 0 and y.min() >= 0 and x.max() < W - 1 and y.max() < H - 1
    ix, iy = x.astype(int), y.astype(int)
    fx, fy = x - ix, y - iy
    a, b, c, d = (image[iy + j, ix + k].astype(float) for j in (0, 1) for k in (0, 1))
    value = (a * (1 - fx) + b * fx) * (1 - fy) + (c * (1 - fx) + d * fx) * fy
    levels = [value[white == w].mean() for w in (False, True)]
    r = value - np.where(white, levels[1], levels[0])
    return 0.5 * (r * r).sum()


def refine(image, quad, template, samples, iterations):
    im, te = torch.from_numpy(image[None]).cuda(), torch.from_numpy(template[None]).cuda()
    co = torch.tensor([quad], dtype=torch.float32, device="cuda")
    loss = torch.full((1,), -1.0, device="cuda")
    args = bdcudatag.refine_args(im, co, te, None, None, samples)
    assert bdcudatag.lib().bd_refine_gauss_newton(args, co.data_ptr(), iterations, loss.data_ptr(), None) == 0
    return co.cpu().numpy()[0].astype(float), float(loss)


@pytest.mark.parametrize("iterations", [0, 1, 2])
@pytest.mark.parametrize("low,high", [(100, 140), (120, 124), (120, 121)])
@pytest.mark.parametrize("cells,samples", [(8, 4), (10, 8), (16, 16)])
def test_low_contrast(cells, samples, low, high, iterations):
    rng = np.random.default_rng(cells + low)
    template = rng.integers(0, 2, (cells, cells)).astype(np.uint8)
    template[0, 0], template[1, 1] = 0, 1
    image = rng.integers(low, high + 1, (H, W)).astype(np.uint8)
    corners, loss = refine(image, [60.3, 50.2, 200.7, 61.1, 190.4, 180.9, 70.8, 170.5], template, samples, iterations)
    want = loss64(image, corners, template, samples)
    assert abs(loss - want) <= 2e-5 * want


def square(at, side):
    return [at, at, at + side, at, at + side, at + side, at, at + side]


def test_cells_of_one_value():
    """16-pixel cells of alternating columns, sampled every 4 pixels at one phase:
    120.3 and 134.6 everywhere, no residual."""
    rng = np.random.default_rng(3)
    template = rng.integers(0, 2, (10, 10)).astype(np.uint8)
    white = np.kron(template, np.ones((16, 16), np.uint8))
    columns = np.arange(160) % 2
    image = np.full((H, W), 120, np.uint8)
    image[24:184, 24:184] = np.where(white, 134 + 2 * columns, 120 + columns)
    corners, loss = refine(image, square(40.3, 128.0), template, 4, 0)
    assert np.array_equal(corners, np.float32(square(40.3, 128.0)))
    assert 0.0 <= loss <= 5e-9 * 1600


@pytest.mark.parametrize("iterations", [1, 2, 3])
@pytest.mark.parametrize("offset", [0.6, 0.9, 1.2])
def test_levels_moved_by_a_step(offset, iterations):
    """Edges are ramps of 3 pixels and samples lie 2 pixels from them: on the
    tag no sample is in a ramp; off it a few are, and shift the levels."""
    template = np.zeros((10, 10), np.uint8)
    template[:, 1::3] = 1
    template[0, 0] = 1
    ramps = np.pad(np.kron(template, np.ones((16, 16))) * 246.0 + 3.0, 8, mode="edge")
    for axis in (0, 1):
        ramps = sum(np.roll(ramps, k, axis) for k in (-1, 0, 1)) / 3
    image = np.full((H, W), 3, np.uint8)
    image[26:202, 26:202] = np.round(ramps)
    corners, loss = refine(image, square(49.5 + offset, 128.0), template, 4, iterations)
    want = loss64(image, corners, template, 4)
    n, e = 1600, 8.4e-4
    assert abs(loss - want) <= e * np.sqrt(2 * n * want) + n * e * e / 2
