"""FP64 grid and median blur at the edges of their tiles, against the oracle (bit-exact)."""
import numpy as np
import pytest

from conftest import same_bits
from oracle import blur, raster

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('xsize,ysize', [(1, 1), (1, 33), (31, 32), (32, 32), (33, 31), (64, 1), (65, 97)])
def test_grid_at_tile_edges(xsize, ysize):
    from vissatsatellitestereo_gb300.proj_to_grid import proj_to_grid
    rng = np.random.default_rng(xsize * 100 + ysize)
    n = int(0.7 * xsize * ysize) + 1                     # sparse: holes with 0 to 8 valid neighbours
    args = (354052.25, 6182702.5, 0.5, 0.5, xsize, ysize)
    p = np.stack([354052.25 + rng.uniform(-0.5, xsize * 0.5 + 0.5, n), 6182702.5 - rng.uniform(-0.5, ysize * 0.5 + 0.5, n),
                  rng.choice([0.0, -0.0, 3.25, -7.5, np.nan, 12.125], n)], axis=1)
    assert same_bits(proj_to_grid(p, *args), raster.proj_to_grid(p, *args))


@pytest.mark.parametrize('H,W', [(1, 30), (1, 61), (61, 1), (2, 31), (7, 29), (8, 30), (9, 31), (16, 60), (17, 61), (33, 92)])
def test_blur_at_strip_edges(H, W):
    from vissatsatellitestereo_gb300.proj_to_grid import median_blur3x3
    rng = np.random.default_rng(H * 100 + W)
    img = rng.normal(0.0, 5.0, (3, H, W)).astype(np.float32)
    img[1][rng.random((H, W)) < 0.05] = np.nan           # windows with and without NaN and zeros
    img[1][rng.random((H, W)) < 0.05] = np.float32(-0.0)
    img[1][rng.random((H, W)) < 0.05] = np.float32(0.0)
    img[2][rng.random((H, W)) < 0.2] = np.inf
    for a in (img, img.astype(np.float64) * (1.0 + 1e-9)):
        got = median_blur3x3(a)
        for b in range(3):
            assert same_bits(got[b], blur.median_blur3x3(a[b].astype(np.float32)))
