"""Bands of frames around 4,096 pixels, where the threads of k_merge change (gpu): as
test_gpu_band_threads, at the bound and at the widest frame."""
import pytest

from test_gpu_band_threads import test_bands as check_bands

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("band_cap", [256, 2048])
@pytest.mark.parametrize("w,h,count", [(4096, 45, 3), (4097, 45, 3), (8192, 40, 3), (4097, 45, 64)])
def test_wide_bands(w, h, count, band_cap):
    check_bands(w, h, count, band_cap)
