"""Batched tiles at the edges of their pixel units: rows that start anywhere within 16 bytes, maps
narrower than a unit, pixels far larger than the grid, pixels on every cell boundary, and
fills from neighbours of very different size.  Bit-exact against the oracle."""
import numpy as np
import pytest
import torch

from conftest import same_bits
from oracle import maps as omaps

pytestmark = pytest.mark.gpu


def _run(spec, m, affine, tile, start, pad):
    from vissatsatellitestereo_gb300.batch import AoiBatch, AoiGrid, MapAffine, MapView
    H, W = m.shape
    buf = np.full(start + H * (W + pad), 9.0, dtype=np.float32)
    buf[start:].reshape(H, W + pad)[:, :W] = m
    store = torch.from_numpy(buf).cuda()[start:].view(H, W + pad)
    b = AoiBatch([AoiGrid(spec.xoff, spec.yoff, spec.res, spec.res, spec.xsize, spec.ysize)],
                 [[MapView(store, W, H, MapAffine(**affine))]], tile=tile)
    vd = b.new_view_dsm()
    b.run(vd)
    got = b.view_dsm(vd, 0).cpu().numpy()
    b.close()
    g = {'xoff': spec.xoff, 'yoff': spec.yoff, 'xres': spec.res, 'yres': spec.res, 'xsize': spec.xsize, 'ysize': spec.ysize}
    assert same_bits(got, omaps.view_dsm(m, affine, g))


def _heights(rng, H, W, wide):
    if wide:          # exponents 30 apart and subnormals among the neighbours of a fill
        m = rng.normal(0.0, 1.0, (H, W)) * rng.choice([1e-42, 1e-30, 1e-4, 1.0, 1e5, 1e30, 3e38], (H, W))
        m = np.clip(m, -3.4e38, 3.4e38)
    else:
        m = rng.normal(5.0, 3.0, (H, W))
    m = m.astype(np.float32)
    m[rng.random((H, W)) < 0.25] = np.nan
    return m


@pytest.mark.parametrize('W', [1, 3, 7, 8, 9, 17, 130])
@pytest.mark.parametrize('start,pad', [(0, 0), (1, 0), (2, 5), (3, 2)])
def test_units_at_any_alignment(W, start, pad):
    from vissatsatellitestereo_gb300 import synth
    rng = np.random.default_rng(100 * W + start)
    s = synth.AoiSpec(0, 354052.25, 6182702.5, 0.5, 67, 131, 1, 0, 1)
    m = _heights(rng, 121, W, wide=W % 2 == 1)
    _run(s, m, synth.map_affine(s.xoff + 16.0, s.yoff - 33.0, 0.52, 0.02 * start), 64 if W % 2 else 32, start, pad)


# up to 15.9 m: the map's steps are 32-bit in units of 2^-28 m and half a pixel
@pytest.mark.parametrize('cells_x,cells_y', [(70, 66), (11, 9), (1, 1), (200, 3)])
@pytest.mark.parametrize('gsd,theta', [(15.9, 0.3), (9.0, -2.0), (1.7, 1.0), (0.003, 0.1)])
def test_pixels_of_any_size(gsd, theta, cells_x, cells_y):
    from vissatsatellitestereo_gb300 import synth
    rng = np.random.default_rng(int(gsd) + 1)
    s = synth.AoiSpec(0, 354052.25, 6182702.5, 0.5, cells_x, cells_y, 1, 0, 1)
    m = _heights(rng, 45, 53, wide=False)
    _run(s, m, synth.map_affine(s.xoff + 0.25 * cells_x, s.yoff - 0.25 * cells_y, gsd, theta), 64, 1, 1)


@pytest.mark.parametrize('shift', [0.0, 0.125, 0.25])
def test_pixels_on_every_cell_boundary(shift):
    from vissatsatellitestereo_gb300 import synth
    rng = np.random.default_rng(3)
    s = synth.AoiSpec(0, 354052.25, 6182702.5, 0.25, 90, 77, 1, 0, 1)
    m = _heights(rng, 100, 111, wide=True)
    _run(s, m, synth.map_affine(s.xoff + 12.0 + shift, s.yoff - 10.0 - shift, 0.25, 0.0), 32, 3, 0)
