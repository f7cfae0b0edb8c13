"""Grids of more rows than a launch holds tiles along y (65,535 tiles of 32 rows), against the
oracle (bit-exact)."""
import numpy as np
import pytest

from conftest import same_bits
from oracle import blur, raster

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


def test_dsm_of_many_rows(cloud, grid):
    import torch
    from vissatsatellitestereo_gb300.produce_dsm import dsm_from_points
    want = blur.median_blur3x3(grid.astype(np.float32))
    args = (XOFF, YOFF, RES, RES, XSIZE, YSIZE)
    pts = torch.from_numpy(cloud).cuda()
    offs = np.array([0, len(cloud)])
    for got in (dsm_from_points(pts, offs, *args), dsm_from_points(pts, offs, *args, epilogue_stream=torch.cuda.Stream()),
                dsm_from_points(pts, offs, *args, pipelined=True), dsm_from_points(cloud, offs, *args)):
        assert same_bits(got[0].cpu().numpy(), want)


def test_depth_maps_onto_many_rows():
    """The AOI's heights lie in the last rows of the grid: the fused form against the points path."""
    import torch
    from oracle import geo
    from vissatsatellitestereo_gb300 import synth
    from vissatsatellitestereo_gb300.aggregate_2p5d_util import depth_map_to_points, dsm_from_depth_maps
    from vissatsatellitestereo_gb300.produce_dsm import dsm_from_points

    def utm(la, lo, z, s):
        e, n = geo.geodetic_to_utm(np.array([la]), np.array([lo]), z, s)
        return float(e[0]), float(n[0])
    case = synth.make_depth_case(61, 1, 150, 190, utm, aoi_m=100.0, lat0=41.0, n_boxes=10)
    aoi, depth = case.aoi, synth.depth_map_torch(case, 0, 'cuda')
    zone = (aoi['zone_number'], aoi['hemisphere'] == 'S')
    args = (aoi['ul_easting'] + 50.0, aoi['ul_northing'] + (YSIZE - 300) * RES, RES, RES, XSIZE, YSIZE)
    fused = dsm_from_depth_maps([depth], list(case.inv_proj), aoi, args, 'fast', [zone]).cpu().numpy()
    pts = depth_map_to_points(depth, case.inv_proj[0], aoi, 'fast', *zone)
    want = dsm_from_points(pts, np.array([0, pts.shape[0]]), *args).cpu().numpy()
    assert same_bits(fused, want) and np.isfinite(fused[0, -1]).any()
