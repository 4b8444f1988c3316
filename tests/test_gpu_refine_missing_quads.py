"""Quads that are not there (gpu): corners that are not numbers, infinite or far outside
beside one ordinary quad.  No sample of them lies in the frame: residuals, losses
and gradients are 0, Gauss-Newton leaves the corners as they are, and the
ordinary quad's results are those that it has alone.  All exact.
"""
import numpy as np
import pytest

import bdcudatag

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

NAN, INF = float("nan"), float("inf")
QUAD = [60.3, 50.2, 200.7, 61.1, 190.4, 180.9, 70.8, 170.5]
MISSING = {
    "nan": [NAN] * 8,
    "one nan": QUAD[:5] + [NAN] + QUAD[6:],
    "infinite": [INF] * 8,
    "one infinite": [5.0, 5.0, INF, 5.0, 50.0, 50.0, 5.0, 50.0],
    "overflow": [3e38, 10.0, -3e38, 10.0, 50.0, 60.0, 10.0, 60.5],
    "overflow, no area": [3e38, 10.0, -3e38, 10.0, 50.0, 60.0, 10.0, 60.0],
    "far left": [-1e10, -1e10, -9e9, -1e10, -9e9, -9e9, -1e10, -9e9],
    "far right": [1e10, 1e10, 1.1e10, 1e10, 1.1e10, 1.1e10, 1e10, 1.1e10],
}


def scene(corners):
    rng = np.random.default_rng(4)
    n = len(corners)
    image = torch.from_numpy(rng.integers(0, 256, (1, 240, 320)).astype(np.uint8)).cuda()
    templates = torch.from_numpy(np.stack([bdcudatag.tag_template(0, 7)] * n)).cuda()
    return image, torch.tensor(corners, dtype=torch.float32, device="cuda"), templates


def gradients(corners):
    image, co, templates = scene(corners)
    levels = torch.tensor([[30.0, 220.0]] * len(corners), device="cuda")
    res = torch.full((len(corners), 6400), -1.0, device="cuda")
    loss, gc = torch.full((len(corners),), -1.0, device="cuda"), torch.full((len(corners), 8), -1.0, device="cuda")
    args = bdcudatag.refine_args(image, co, templates, None, levels, 8)
    assert bdcudatag.lib().bd_refine_forward(args, res.data_ptr(), loss.data_ptr(), None) == 0
    torch.cuda.synchronize()
    ones = torch.ones_like(res)
    assert bdcudatag.lib().bd_refine_backward(args, ones.data_ptr(), gc.data_ptr(), None, None) == 0
    torch.cuda.synchronize()
    return [t.cpu().numpy() for t in (res, loss, gc)]


def gauss_newton(corners):
    image, co, templates = scene(corners)
    loss = torch.full((len(corners),), -1.0, device="cuda")
    args = bdcudatag.refine_args(image, co, templates, None, None, 8)
    assert bdcudatag.lib().bd_refine_gauss_newton(args, co.data_ptr(), 3, loss.data_ptr(), None) == 0
    torch.cuda.synchronize()
    return co.cpu().numpy(), loss.cpu().numpy()


@pytest.mark.parametrize("name", MISSING)
def test_residuals_and_adjoint(name):
    both, alone = gradients([MISSING[name], QUAD]), gradients([QUAD])
    for got, want in zip(both, alone):
        assert np.all(got[0] == 0.0)
        assert np.array_equal(got[1], want[0])


@pytest.mark.parametrize("name", MISSING)
def test_gauss_newton(name):
    (corners, loss), (want, want_loss) = gauss_newton([MISSING[name], QUAD]), gauss_newton([QUAD])
    assert np.array_equal(corners[0], np.float32(MISSING[name]), equal_nan=True)
    assert loss[0] == 0.0
    assert np.array_equal(corners[1], want[0]) and loss[1] == want_loss[0]
