"""Per-view DSMs at the edges of the epilogue's 64 x 32 tiles, in every form of the call, against the
oracle's proj_to_grid and blur (bit-exact): borders inside and at the ends of tiles, uncovered
parts, zeros of both signs."""
import numpy as np
import pytest
import torch

from conftest import same_bits
from oracle import blur, raster

pytestmark = pytest.mark.gpu


def _cloud(xsize, ysize, view, rng):
    n = int((1.5 + view) * xsize * ysize) + 3
    e = 354052.25 + rng.uniform(-0.5, xsize * 0.5 + 0.5, n)
    s = rng.uniform(-0.5, ysize * 0.5 * (0.6 if view == 1 else 1.0) + 0.5, n)        # view 1: a part is uncovered
    z = rng.normal(20.0, 5.0, n)
    if view == 2:
        z = rng.choice([0.0, -0.0, 4.5, -3.0, np.nan], n)
    return np.stack([e, 6182702.5 - s, z], axis=1)


@pytest.mark.parametrize('xsize,ysize', [(1, 1), (1, 40), (70, 1), (2, 33), (63, 31), (64, 32), (65, 33), (66, 34), (127, 65),
                                         (130, 64)])
def test_dsm_at_tile_edges(xsize, ysize):
    from vissatsatellitestereo_gb300.produce_dsm import dsm_from_points
    rng = np.random.default_rng(xsize * 1000 + ysize)
    clouds = [_cloud(xsize, ysize, v, rng) for v in range(3)]
    args = (354052.25, 6182702.5, 0.5, 0.5, xsize, ysize)
    want = [blur.median_blur3x3(raster.proj_to_grid(c, *args).astype(np.float32)) for c in clouds]
    pts = torch.from_numpy(np.concatenate(clouds)).cuda()
    offs = np.cumsum([0] + [len(c) for c in clouds])
    epi = torch.cuda.Stream()
    forms = (dsm_from_points(pts, offs, *args), dsm_from_points(pts, offs, *args, pipelined=True),
             dsm_from_points(pts, offs, *args, epilogue_stream=epi), dsm_from_points(np.concatenate(clouds), offs, *args))
    for got in forms:
        for v in range(3):
            assert same_bits(got[v].cpu().numpy(), want[v]), v


@pytest.mark.parametrize('tile', [32, 64])
@pytest.mark.parametrize('xsize,ysize', [(1, 1), (1, 70), (70, 1), (31, 33), (32, 32), (33, 31), (63, 65), (64, 64), (65, 63),
                                         (66, 130)])
def test_batched_tiles_at_their_edges(tile, xsize, ysize):
    from vissatsatellitestereo_gb300 import synth
    from vissatsatellitestereo_gb300.batch import AoiBatch, AoiGrid, MapAffine, MapView, map_points
    rng = np.random.default_rng(tile + xsize * 1000 + ysize)
    spec = synth.AoiSpec(0, 354052.25, 6182702.5, 0.5, xsize, ysize, 2, 0, 7)
    h, w = int(1.3 * ysize) + 3, int(1.2 * xsize) + 3
    affs = synth.aoi_view_affines(spec, width=w, height=h)
    maps = [torch.from_numpy(rng.normal(10.0, 4.0, (h, w)).astype(np.float32)).cuda() for _ in range(2)]
    for m in maps:
        m[torch.from_numpy(rng.random((h, w)) < 0.25).cuda()] = float('nan')
    maps[1][torch.from_numpy(rng.random((h, w)) < 0.2).cuda()] = -0.0
    b = AoiBatch([AoiGrid(spec.xoff, spec.yoff, 0.5, 0.5, xsize, ysize)],
                 [[MapView(m, w, h, MapAffine(**a)) for m, a in zip(maps, affs)]], tile=tile)
    buf = b.run(b.new_view_dsm())
    for v in range(2):
        pts = map_points(maps[v], affs[v]).cpu().numpy()
        want = blur.median_blur3x3(raster.proj_to_grid(pts, spec.xoff, spec.yoff, 0.5, 0.5, xsize, ysize).astype(np.float32))
        assert same_bits(b.view_dsm(buf, v).cpu().numpy(), want), v
