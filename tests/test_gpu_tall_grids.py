"""Grids of more rows than a launch holds tiles along y (65,535 tiles of 32 rows), against the
oracle (bit-exact)."""
import numpy as np
import pytest

from conftest import same_bits
from oracle import raster

pytestmark = pytest.mark.gpu

XOFF, YOFF, RES, XSIZE, YSIZE = 354052.25, 7182702.5, 0.25, 2, 65535 * 32 + 1


@pytest.fixture(scope='module')
def cloud():
    """One point in almost every cell, the last row's among them: a few holes."""
    rng = np.random.default_rng(11)
    row, col = (a.ravel() for a in np.meshgrid(np.arange(YSIZE), np.arange(XSIZE), indexing='ij'))
    kept = rng.random(row.size) > 0.02
    row, col = row[kept], col[kept]
    u = rng.uniform(0.1, 0.9, (2, row.size))
    return np.stack([XOFF + (col + u[0]) * RES, YOFF - (row + u[1]) * RES, rng.normal(20.0, 5.0, row.size)], axis=1)


@pytest.fixture(scope='module')
def grid(cloud):
    want = raster.proj_to_grid(cloud, XOFF, YOFF, RES, RES, XSIZE, YSIZE)
    assert np.isfinite(want[-1]).all()
    return want


def test_proj_to_grid_of_many_rows(cloud, grid):
    from vissatsatellitestereo_gb300.proj_to_grid import proj_to_grid
    assert same_bits(proj_to_grid(cloud, XOFF, YOFF, RES, RES, XSIZE, YSIZE), grid)
