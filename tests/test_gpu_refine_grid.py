"""Residuals and adjoint over every shape of the sample grid (gpu): side lengths
below, at and above a warp's block of 8 columns and the warps' ten blocks, against the
same in 64 bits.

Tolerance: a sample's position carries 3e-5 px of FP32 rounding near 300 px, a
gradient of this texture is below 60 DN/px, so a residual is within 4e-3 DN; the
gradients are sums of products of such values with relative errors of 1e-4 a term
at most, and lie within 1e-3 of their norm.
"""
import numpy as np
import pytest

import bdcudatag
from test_gpu_refine import S, ref_forward  # noqa: F401  (the FP64 restatement's sample rule)
import test_gpu_refine

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

W, H = 320, 240


@pytest.mark.parametrize("cells,samples", [(4, 1), (4, 3), (8, 2), (5, 5), (8, 8), (10, 8), (11, 8), (16, 5), (16, 16)])
def test_grid(cells, samples, monkeypatch):
    monkeypatch.setattr(test_gpu_refine, "S", samples)
    rng = np.random.default_rng(100 * cells + samples)
    noise = np.kron(rng.uniform(0, 255, (H // 8 + 2, W // 8 + 2)), np.ones((8, 8)))
    smooth = sum(noise[j:j + H, i:i + W] for j in range(8) for i in range(8)) / 64
    base = np.array([[60.3, 50.2], [200.7, 61.1], [190.4, 180.9], [70.8, 170.5]])
    quads = np.stack([base, base[::-1] * 0.9 + 7, base + [150.0, 90.0]]).reshape(3, 8).astype(np.float32)
    im = torch.from_numpy(np.stack([smooth, smooth.T[:H, :H].repeat(2, 1)[:, :W]]).astype(np.uint8)).cuda()
    co = torch.from_numpy(quads).cuda()
    te = torch.from_numpy(rng.integers(0, 2, (3, cells, cells)).astype(np.uint8)).cuda()
    ix = torch.tensor([0, 1, 0], dtype=torch.int32, device="cuda")
    lv = torch.from_numpy(np.tile(np.array([[40.0, 200.0]], np.float32), (3, 1))).cuda()
    n = (cells * samples) ** 2
    res, loss = torch.full((3, n), -1.0, device="cuda"), torch.empty(3, device="cuda")
    gc, gi = torch.empty((3, 8), device="cuda"), torch.zeros(im.shape, device="cuda")
    args = bdcudatag.refine_args(im, co, te, ix, lv, samples)
    assert bdcudatag.lib().bd_refine_forward(args, res.data_ptr(), loss.data_ptr(), None) == 0
    assert bdcudatag.lib().bd_refine_backward(args, res.data_ptr(), gc.data_ptr(), gi.data_ptr(), None) == 0
    c64, i64 = co.double().requires_grad_(True), im.double().requires_grad_(True)
    r64, l64 = ref_forward(i64, c64, te, ix, lv.double())
    l64.sum().backward()
    assert (res.double() - r64).abs().max() < 4e-3
    assert torch.allclose(loss.double(), l64, rtol=1e-4)
    assert (gc.double() - c64.grad).norm() < 1e-3 * c64.grad.norm()
    assert (gi.double() - i64.grad).norm() < 1e-3 * i64.grad.norm()
