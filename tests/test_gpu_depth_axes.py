"""Fused depth-map binning against the points path (bit-exact) over frames whose grid origins lie
in different binades: the fixed-point axes (2^10 .. 2^23) and the ones beside them, and points
far from the grid in either direction."""
import numpy as np
import pytest
import torch

from conftest import same_bits
from oracle import geo

pytestmark = pytest.mark.gpu


def _utm(la, lo, z, s):
    e, n = geo.geodetic_to_utm(np.array([la]), np.array([lo]), z, s)
    return float(e[0]), float(n[0])


def test_fixed_point_difference_is_the_bit_pattern_difference():
    """((E + 1022) << 52) + (S << (22 - E)) is the pattern of S 2^-30 in the binade 2^E."""
    rng = np.random.default_rng(0)
    for e in range(10, 23):
        s = np.concatenate([rng.integers(1 << (e + 30), 1 << (e + 31), 2000), [1 << (e + 30), (1 << (e + 31)) - 1]])
        bits = (s.astype(np.float64) * 2.0**-30).view(np.int64)
        assert np.array_equal(bits, ((e + 1022) << 52) + (s << (22 - e)))


@pytest.mark.parametrize('lat,lon,shift', [
    (0.02, 9.0, 0.0),              # northing of a few km
    (2.0, 10.5, 0.0),              # 2^17
    (39.77, -84.05, 0.0),          # 2^22: the usual case
    (75.9, 20.0, 0.0),             # above 2^23: northing through its double
    (-0.05, 9.0, 0.0),             # false northing near 10,000 km
    (39.77, -84.05, 4.0e5),        # grid far east of every point
    (39.77, -84.05, -7.3e5),       # grid origin at an easting of a few km
])
def test_fused_binning_equals_the_points_path(lat, lon, shift):
    from vissatsatellitestereo_gb300 import synth
    from vissatsatellitestereo_gb300.aggregate_2p5d_util import depth_map_to_points, dsm_from_depth_maps
    from vissatsatellitestereo_gb300.produce_dsm import dsm_from_points
    case = synth.make_depth_case(51, 2, 150, 190, _utm, aoi_m=200.0, lat0=lat, lon0=lon, n_boxes=20)
    aoi = case.aoi
    zones = [(aoi['zone_number'], aoi['hemisphere'] == 'S')] * 2
    xoff = aoi['ul_easting'] + shift
    for dx in (0.0, 0.25):
        if xoff + dx <= 0:
            xoff = 1500.0
        grid = (xoff + dx, aoi['ul_northing'] - dx, 0.5, 0.5, 400, 390)
        depths = [synth.depth_map_torch(case, v, 'cuda') for v in range(2)]
        fused = dsm_from_depth_maps(depths, list(case.inv_proj), aoi, grid, 'fast', zones).cpu().numpy()
        pts = [depth_map_to_points(d, case.inv_proj[v], aoi, 'fast', *zones[v]) for v, d in enumerate(depths)]
        offs = torch.tensor(np.cumsum([0] + [p.shape[0] for p in pts]), dtype=torch.int64, device='cuda')
        want = dsm_from_points(torch.cat(pts), offs, *grid).cpu().numpy()
        assert same_bits(fused, want)
        if shift == 0.0:
            assert np.isfinite(fused).any()
