"""Images and grids of a few columns or rows, alone and in stacks, on both sides of the rules that give them a
thread per cell or long tiles, against the oracle (bit-exact)."""
import numpy as np
import pytest

from conftest import same_bits
from oracle import blur, raster

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n,H,W', [(700, 1, 1), (5, 1, 2), (300, 3, 3), (90, 6, 6), (2, 1000, 1), (3, 257, 2), (2, 300, 5),
                                   (2, 300, 6), (2, 1, 700), (2, 2, 300), (40, 9, 3), (1, 4099, 4)])
def test_blur_of_narrow_images(n, H, W):
    from vissatsatellitestereo_gb300.proj_to_grid import median_blur3x3
    rng = np.random.default_rng(n + H * 100 + W)
    img = rng.normal(0.0, 5.0, (n, H, W)).astype(np.float32)
    u = rng.random((n, H, W))
    for k, v in enumerate((np.nan, np.inf, 0.0, -0.0)):
        img[1::2][(u[1::2] >= 0.06 * k) & (u[1::2] < 0.06 * (k + 1))] = v      # every other image: clean
    for a in (img, img.astype(np.float64) * (1.0 + 1e-9)):
        got = median_blur3x3(a)
        for b in range(n):
            assert same_bits(got[b], blur.median_blur3x3(a[b].astype(np.float32))), b


@pytest.mark.parametrize('xsize,ysize', [(1, 700), (2, 1025), (4, 256), (5, 257), (8, 511), (9, 300), (700, 1), (1025, 2),
                                         (256, 4), (257, 5), (511, 8), (300, 9)])
def test_grid_of_few_columns_or_rows(xsize, ysize):
    from vissatsatellitestereo_gb300.proj_to_grid import proj_to_grid
    rng = np.random.default_rng(xsize * 100 + ysize)
    n = int(0.7 * xsize * ysize) + 1                     # sparse: holes with 0 to 8 valid neighbours
    args = (354052.25, 6182702.5, 0.5, 0.5, xsize, ysize)
    p = np.stack([354052.25 + rng.uniform(-0.5, xsize * 0.5 + 0.5, n), 6182702.5 - rng.uniform(-0.5, ysize * 0.5 + 0.5, n),
                  rng.choice([0.0, -0.0, 3.25, -7.5, np.nan, 12.125], n)], axis=1)
    assert same_bits(proj_to_grid(p, *args), raster.proj_to_grid(p, *args))
