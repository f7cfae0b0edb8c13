"""The work that users of this framework have it do, as cases that can be timed and compared.

Each case is one call (or the few calls that belong together) of a public entry point, over
the sizes that the repository's own configurations, tests and benchmark use: a handful of
tie points up to a 50-view AOI.  ``prepare`` makes what a program holds before the call (inputs on
the GPU, cameras, a batch plan), ``run`` is one pass, ``exact`` the same outputs from plain
64-bit torch.
"""
import functools
import math
import random

import numpy as np
import torch

from vissatsatellitestereo_gb300 import _lib, synth
from vissatsatellitestereo_gb300.aggregate_2p5d import fuse_dsms
from vissatsatellitestereo_gb300.aggregate_2p5d_util import dsm_from_depth_maps
from vissatsatellitestereo_gb300.batch import AoiBatch, AoiGrid, MapAffine, MapView
from vissatsatellitestereo_gb300.camera_approx import approx_perspective_enu
from vissatsatellitestereo_gb300.coordinate_system import latlon_to_eastnorh
from vissatsatellitestereo_gb300.produce_dsm import dsm_from_points
from vissatsatellitestereo_gb300.proj_to_grid import median_blur3x3, proj_to_grid
from vissatsatellitestereo_gb300.rpc_model import RPCModel, project_cameras, project_cube
from vissatsatellitestereo_gb300.solve_affine import approx_affine_latlonalt

F64 = torch.float64


# --------------------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------------------
def listed():
    return [
        # tie points through one camera: the smallest call
        {'name': 'project_tie_points', 'kind': 'project', 'cams': 1, 'n': 1999, 'mode': 'exact', 'keep': False},
        # a dense cloud of normalised points into every view, as a tensor-core contraction
        {'name': 'project_cube', 'kind': 'cube', 'cams': 50, 'n': 2000000, 'variant': 'bf16x3_lin'},
        # image points back to the ground at given altitudes
        {'name': 'inverse_points', 'kind': 'inverse', 'n': 90001},
        # one camera approximated over a 101 x 101 x 21 grid (one image at a time)
        {'name': 'fit_one_view', 'kind': 'fit', 'views': 1, 'n_xy': 101, 'n_z': 21, 'shared': True, 'mode': 'fast'},
        # all cameras of a 50-view AOI, each over its own 200 x 200 x 20 grid
        {'name': 'fit_aoi', 'kind': 'fit', 'views': 50, 'n_xy': 200, 'n_z': 20, 'shared': False, 'mode': 'fast'},
        # affine cameras of an AOI's views over one shared grid
        {'name': 'affine_aoi', 'kind': 'affine', 'views': 12, 'n_xy': 101, 'n_z': 21},
        # one height map's points onto a 0.5 m grid (FP64 DSM), and its median blur
        {'name': 'grid_one_view', 'kind': 'grid', 'image': 1024, 'cells_x': 1025, 'cells_y': 1025, 'res': 0.5},
        # the point clouds of an AOI's views, of uneven sizes, onto one grid
        {'name': 'dsm_views', 'kind': 'dsm', 'views': 10, 'image': 3001, 'cells_x': 1503, 'cells_y': 1409,
         'res': 0.3},
        # COLMAP depth maps of an AOI straight to per-view DSMs
        {'name': 'depth_views', 'kind': 'depth', 'views': 6, 'height': 2047, 'width': 2300, 'cells': 1201,
         'res': 0.5, 'mode': 'fast', 'zones': True},
        # the 50-view fusion of one AOI
        {'name': 'fuse_views', 'kind': 'fuse', 'views': 50, 'h': 2000, 'w': 2000, 'layout': 'vhw'},
        # a site seen by more views than one season brings, stacked as the reference stacks them
        {'name': 'fuse_many_views', 'kind': 'fuse', 'views': 97, 'h': 409, 'w': 451, 'layout': 'hwv'},
        # many uneven AOIs in one batch: per-view DSMs, then their fusions
        {'name': 'aoi_batch', 'kind': 'batch', 'aois': 8, 'layout': 3, 'image_lo': 512, 'image_hi': 2048,
         'views_lo': 4, 'views_hi': 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['project', 'project', 'cube', 'inverse', 'fit', 'fit', 'affine', 'grid', 'dsm', 'depth', 'fuse',
                       'fuse', 'batch'])
    if kind == 'project':
        cams = _log(rng, 1, 50)
        mode = rng.choice(['exact', 'fast'])
        top = 1000000 if mode == 'fast' else 400000
        return {'kind': kind, 'cams': cams, 'n': _log(rng, 100, max(200, min(1000000, 8 * top // cams))), 'mode': mode,
                'keep': rng.random() < 0.5}
    if kind == 'cube':
        cams = _log(rng, 1, 60)
        return {'kind': kind, 'cams': cams, 'n': _log(rng, 10000, 2000000),
                'variant': rng.choice(['fp32', 'bf16x3_lin', 'bf16x6', 'bf16x3_lin_tc'])}
    if kind == 'inverse':
        return {'kind': kind, 'n': _log(rng, 100, 300000)}
    if kind == 'fit':
        views = _log(rng, 1, 50)
        return {'kind': kind, 'views': views, 'n_xy': _log(rng, 20, 200), 'n_z': _log(rng, 5, 20),
                'shared': rng.random() < 0.5, 'mode': rng.choice(['fast', 'fast', 'exact']) if views < 5 else 'fast'}
    if kind == 'affine':
        return {'kind': kind, 'views': _log(rng, 1, 24), 'n_xy': _log(rng, 20, 101), 'n_z': _log(rng, 5, 21)}
    if kind == 'grid':
        image = _log(rng, 200, 3000)
        res = round(rng.uniform(0.3, 1.0), 2)
        return {'kind': kind, 'image': image, 'cells_x': _log(rng, 0.4 * image, 1.1 * image),
                'cells_y': _log(rng, 0.4 * image, 1.1 * image), 'res': res}
    if kind == 'dsm':
        image = _log(rng, 300, 3000)
        return {'kind': kind, 'views': _log(rng, 1, 12), 'image': image, 'cells_x': _log(rng, 0.3 * image, 1.1 * image),
                'cells_y': _log(rng, 0.3 * image, 1.1 * image), 'res': round(rng.uniform(0.3, 1.0), 2)}
    if kind == 'depth':
        height = _log(rng, 300, 2400)
        return {'kind': kind, 'views': _log(rng, 1, 8), 'height': height,
                'width': int(height * rng.uniform(0.8, 1.3)), 'cells': _log(rng, 300, 1500), 'res': 0.5,
                'mode': 'exact' if height < 700 and rng.random() < 0.3 else 'fast', 'zones': rng.random() < 0.7}
    if kind == 'fuse':
        views = _log(rng, 3, 120)
        side = min(2000.0, math.sqrt(1.5e8 / views if views <= 64 else 2.0e7 / views))
        h = _log(rng, 0.1 * side, side)
        return {'kind': kind, 'views': views, 'h': h, 'w': int(h * rng.uniform(0.7, 1.3)) + 1,
                'layout': rng.choice(['vhw', 'hwv'])}
    lo = _log(rng, 256, 1500)
    vl = rng.randint(3, 12)
    return {'kind': 'batch', 'aois': rng.randint(1, 8), 'layout': rng.randrange(1 << 20), 'image_lo': lo,
            'image_hi': int(lo * rng.uniform(1.0, 1.4)) + 1, 'views_lo': vl, 'views_hi': int(vl * rng.uniform(1.0, 2.0)) + 1}


# --------------------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device='cuda')
    g.manual_seed(int(seed) & 0x7fffffff)
    return g


def _metas(seed, count, image=4096):
    """RPC cameras of one AOI: own coefficients around one shared lat/lon/alt frame."""
    spec = synth.AoiSpec(0, 0.0, 0.0, 0.5, 1, 1, count, image, synth.BASE_SEED + 31 * int(seed))
    return synth.aoi_rpc_metas(spec)


def _cloud(meta, n, seed):
    """n points uniform over the camera's lat/lon/alt box, a little beyond the image."""
    r = meta['rpc']
    u = torch.rand((3, n), generator=_gen(seed), device='cuda', dtype=F64) * 2.1 - 1.05
    return (r['latOff'] + r['latScale'] * u[0], r['lonOff'] + r['lonScale'] * u[1], r['altOff'] + r['altScale'] * u[2])


def _grids(case, metas):
    gs = [synth.rpc_sample_grid_torch(m, case['n_xy'], case['n_z'], 'cuda')
          for m in (metas[:1] if case.get('shared', True) else metas)]
    if case.get('shared', True):
        return gs[0]
    return {k: torch.stack([g[k] for g in gs]) for k in gs[0]}


def _scene(case, seed):
    grid = synth.DsmGrid(synth.EXPLORER_UL_EASTING, synth.EXPLORER_UL_NORTHING, case['res'], case['res'],
                         case['cells_x'], case['cells_y'])
    return synth.make_scene(synth.BASE_SEED + 7 * int(seed), grid, 120, 3.0, 80.0)


def _counts(case):
    """Points kept per view: the clouds' sizes are uneven, as filtering leaves them."""
    rng = random.Random(case['image'] * 1000 + case['views'])
    n = case['image'] ** 2
    return [n - int(n * 0.25 * rng.random()) for _ in range(case['views'])]


def _aoi_specs(case):
    rng = random.Random(case['layout'])
    specs = []
    for a in range(case['aois']):
        img = rng.randint(case['image_lo'], case['image_hi'])
        cells = max(64, int(img * rng.uniform(0.35, 0.8)))
        res = round(rng.uniform(0.3, 1.0), 3)
        xs, ys = cells, int(cells * rng.uniform(0.75, 1.33))
        specs.append(synth.AoiSpec(a, rng.uniform(270000.0, 515000.0 - xs * res), rng.uniform(4200000.0 + ys * res, 8380000.0),
                                   res, xs, ys, rng.randint(case['views_lo'], case['views_hi']), img,
                                   case['layout'] + 7919 * (a + 1)))
    return specs


def _utm(lat, lon, zone, south):
    e, n = latlon_to_eastnorh(np.array([lat]), np.array([lon]))
    return float(e[0]), float(n[0])


def prepare(case, seed):
    kind = case['kind']
    st = {'case': dict(case)}
    if kind == 'project':
        metas = _metas(seed, case['cams'])
        st['metas'] = metas
        if case['cams'] == 1 and not case['keep']:
            st['model'] = RPCModel(metas[0], mode=case['mode'])
        st['points'] = _cloud(metas[0], case['n'], seed + 1)
    elif kind == 'cube':
        st['metas'] = _metas(seed, case['cams'], 4096)
        st['cams'] = torch.from_numpy(_lib.camera_array(st['metas'])).cuda()
        st['xyz'] = torch.rand((3, case['n']), generator=_gen(seed), device='cuda') * 2.0 - 1.0
    elif kind == 'inverse':
        meta = _metas(seed, 1)[0]
        st['meta'], st['model'] = meta, RPCModel(meta)
        g = _gen(seed)
        u = torch.rand((3, case['n']), generator=g, device='cuda', dtype=F64)
        r = meta['rpc']
        st['points'] = (u[0] * meta['width'], u[1] * meta['height'],
                        r['altOff'] + r['altScale'] * (0.4 * u[2] - 0.2))
    elif kind in ('fit', 'affine'):
        st['metas'] = _metas(seed, case['views'])
        st['cams'] = torch.from_numpy(_lib.camera_array(st['metas'])).cuda()
        st['grid'] = _grids(case, st['metas'])
    elif kind == 'grid':
        scene = _scene(case, seed)
        side = case['res'] * max(case['cells_x'], case['cells_y'])
        view = synth.ViewSpec(case['image'], case['image'], side / case['image'], 0.02, 0.0, 0.0, 0.15, 1000 + seed)
        st['points'] = synth.view_points_torch(scene, view, 'cuda')
    elif kind == 'dsm':
        scene = _scene(case, seed)
        views = synth.make_views(synth.BASE_SEED + 12 + seed, scene, case['views'], case['image'], case['image'], 0.10,
                                 0.20, 0.5)
        counts = _counts(case)
        st['points'] = torch.empty((sum(counts), 3), dtype=F64, device='cuda')
        at = 0
        for c, view in zip(counts, views):
            st['points'][at:at + c] = synth.view_points_torch(scene, view, 'cuda')[:c]
            at += c
        st['offsets'] = torch.tensor([0] + np.cumsum(counts).tolist(), dtype=torch.int64, device='cuda')
    elif kind == 'depth':
        side = case['cells'] * case['res']
        dc = synth.make_depth_case(synth.BASE_SEED + 3000 + 17 * seed, case['views'], case['height'], case['width'],
                                   _utm, aoi_m=side, n_boxes=120)
        st['aoi'], st['mats'] = dc.aoi, list(dc.inv_proj)
        st['grid'] = (dc.aoi['ul_easting'], dc.aoi['ul_northing'], case['res'], case['res'], case['cells'], case['cells'])
        st['zones'] = [(dc.aoi['zone_number'], dc.aoi['hemisphere'] == 'S')] * case['views'] if case['zones'] else None
        st['depths'] = [synth.depth_map_torch(dc, v, 'cuda') for v in range(case['views'])]
    elif kind == 'fuse':
        g = _gen(seed)
        v, h, w = case['views'], case['h'], case['w']
        ground = torch.randn((h, w), generator=g, device='cuda') * 10 + 30
        d = ground + torch.randn((v, h, w), generator=g, device='cuda') * 0.4
        for k in range(v):              # per view: a few wrong heights and 10-20% holes
            u = torch.rand((h, w), generator=g, device='cuda')
            d[k] = torch.where(u < 0.05, d[k] + 25.0, d[k])
            d[k][u > 0.80 + 0.1 * ((k * 7) % 11) / 10.0] = float('nan')
        st['dsms'] = d if case['layout'] == 'vhw' else d.permute(1, 2, 0).contiguous()
    elif kind == 'batch':
        specs = _aoi_specs(case)
        pool = synth.height_map_pool(6, max(s.image for s in specs), synth.BASE_SEED + 13 * seed, 'cuda', n_boxes=80)
        affs, views, k = [], [], 0
        for s in specs:
            af = synth.aoi_view_affines(s)
            affs.append(af)
            views.append([MapView(pool[(k + v) % 6], s.image, s.image, MapAffine(**a)) for v, a in enumerate(af)])
            k += s.n_views
        st['specs'], st['pool'], st['affines'] = specs, pool, affs
        b = AoiBatch([AoiGrid(s.xoff, s.yoff, s.res, s.res, s.xsize, s.ysize) for s in specs], views)
        st['batch'], st['view_dsm'], st['fused'], st['scratch'] = b, b.new_view_dsm(), b.new_fused(), b.new_scratch()
    else:
        raise ValueError(kind)
    return st


# --------------------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------------------
def run(st):
    case = st['case']
    kind = case['kind']
    if kind == 'project':
        if 'model' in st:
            return st['model'].projection(*st['points'])
        return project_cameras(st['metas'], *st['points'], mode=case['mode'], keep=case['keep'])
    if kind == 'cube':
        return project_cube(st['cams'], st['xyz'], case['variant'])
    if kind == 'inverse':
        return st['model'].inverse_projection(*st['points'])
    if kind == 'fit':
        g = st['grid']
        return approx_perspective_enu(st['cams'], g['lat'], g['lon'], g['alt'], g['x'], g['y'], g['z'], mode=case['mode'],
                                      shared_points=case['shared'])
    if kind == 'affine':
        g = st['grid']
        return approx_affine_latlonalt(st['cams'], g['lat'], g['lon'], g['alt'])
    if kind == 'grid':
        d = proj_to_grid(st['points'], synth.EXPLORER_UL_EASTING, synth.EXPLORER_UL_NORTHING, case['res'], case['res'],
                         case['cells_x'], case['cells_y'])
        return d, median_blur3x3(d)
    if kind == 'dsm':
        return dsm_from_points(st['points'], st['offsets'], synth.EXPLORER_UL_EASTING, synth.EXPLORER_UL_NORTHING,
                               case['res'], case['res'], case['cells_x'], case['cells_y'])
    if kind == 'depth':
        return dsm_from_depth_maps(st['depths'], st['mats'], st['aoi'], grid=st['grid'], mode=case['mode'],
                                   zones=st['zones'])
    if kind == 'fuse':
        return fuse_dsms(st['dsms'], layout=case['layout'])
    b = st['batch']
    b.run(st['view_dsm'])
    return b.fuse(st['view_dsm'], st['fused'], st['scratch']), st['view_dsm']


# --------------------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------------------
def work(case):
    kind = case['kind']
    if kind == 'project':            # 4 cubic polynomials of 20 terms, two quotients, denormalisation
        out = 17 if case['keep'] else 16
        return {'bytes': 24 * case['n'] + out * case['n'] * case['cams'], 'flops': 270 * case['n'] * case['cams']}
    if kind == 'cube':
        return {'bytes': 12 * case['n'] + 8 * case['n'] * case['cams'], 'flops': 166 * case['n'] * case['cams']}
    if kind == 'inverse':            # about eight iterations of three projections and an update
        return {'bytes': 48 * case['n'], 'flops': 8 * 800 * case['n']}
    if kind == 'fit':                # projection, moments, residuals
        n = case['n_xy'] ** 2 * case['n_z']
        sets = 1 if case['shared'] else case['views']
        return {'bytes': 48 * n * sets + 8 * 20 * case['views'], 'flops': 450 * n * case['views']}
    if kind == 'affine':
        n = case['n_xy'] ** 2 * case['n_z']
        return {'bytes': 24 * n + 80 * case['views'], 'flops': 320 * n * case['views']}
    if kind == 'grid':
        cells = case['cells_x'] * case['cells_y']
        return {'bytes': 24 * case['image'] ** 2 + 12 * cells, 'flops': 6 * case['image'] ** 2 + 40 * cells}
    if kind == 'dsm':
        n, cells = sum(_counts(case)), case['cells_x'] * case['cells_y']
        return {'bytes': 24 * n + 4 * cells * case['views'], 'flops': 6 * n + 40 * cells * case['views']}
    if kind == 'depth':              # homogeneous divide, ENU -> geodetic -> UTM, binning
        n, cells = case['views'] * case['height'] * case['width'], case['views'] * case['cells'] ** 2
        return {'bytes': 4 * n + 4 * cells, 'flops': 150 * n + 40 * cells}
    if kind == 'fuse':
        cells = case['h'] * case['w']
        return {'bytes': 4 * cells * (case['views'] + 1), 'flops': cells * case['views'] * 20}
    specs = _aoi_specs(case)
    px = sum(s.n_views * s.image ** 2 for s in specs)
    cv = sum(s.n_views * s.cells for s in specs)
    return {'bytes': 4 * px + 4 * cv + 4 * cv + 4 * sum(s.cells for s in specs), 'flops': 6 * px + 60 * cv}


# --------------------------------------------------------------------------------------
# the same outputs in plain 64-bit torch
# --------------------------------------------------------------------------------------
def _poly(c, x, y, z):
    return (c[0] + c[1] * y + c[2] * x + c[3] * z + c[4] * y * x + c[5] * y * z + c[6] * x * z + c[7] * y * y
            + c[8] * x * x + c[9] * z * z + c[10] * x * y * z + c[11] * y * y * y + c[12] * y * x * x + c[13] * y * z * z
            + c[14] * y * y * x + c[15] * x * x * x + c[16] * x * z * z + c[17] * y * y * z + c[18] * x * x * z
            + c[19] * z * z * z)


def _rfm(r, x, y, z):
    return (_poly(r['colNum'], x, y, z) / _poly(r['colDen'], x, y, z),
            _poly(r['rowNum'], x, y, z) / _poly(r['rowDen'], x, y, z))


def _project(meta, lat, lon, alt):
    r = meta['rpc']
    x, y, z = ((lat - r['latOff']) / r['latScale'], (lon - r['lonOff']) / r['lonScale'],
               (alt - r['altOff']) / r['altScale'])
    c, w = _rfm(r, x, y, z)
    return c * r['colScale'] + r['colOff'], w * r['rowScale'] + r['rowOff']


def _inside(meta, col, row):
    return (col >= 0) & (row >= 0) & (col < meta['width']) & (row < meta['height'])


def _exact_inverse(meta, col, row, alt):
    """Newton's method on the normalised projection, far past its rounding."""
    r = meta['rpc']
    c, w, z = (col - r['colOff']) / r['colScale'], (row - r['rowOff']) / r['rowScale'], (alt - r['altOff']) / r['altScale']
    x, y, h = torch.zeros_like(c), torch.zeros_like(c), 1e-5
    for _ in range(30):
        c0, w0 = _rfm(r, x, y, z)
        cx, wx = _rfm(r, x + h, y, z)
        cy, wy = _rfm(r, x, y + h, z)
        a, b, d, e = (cx - c0) / h, (cy - c0) / h, (wx - w0) / h, (wy - w0) / h
        det = a * e - b * d
        x, y = x + (e * (c - c0) - b * (w - w0)) / det, y + (a * (w - w0) - d * (c - c0)) / det
    return y * r['lonScale'] + r['lonOff'], x * r['latScale'] + r['latOff'], alt


def _exact_fit(meta, g):
    """The unit camera vector with the smallest DLT residual, its factors and its errors."""
    col, row = _project(meta, g['lat'], g['lon'], g['alt'])
    k = _inside(meta, col, row)
    c, w = col[k], row[k]
    X = torch.stack([g['x'][k], g['y'][k], g['z'][k]], 1)
    mid, s = (X.amax(0) + X.amin(0)) / 2, float((X.amax(0) - X.amin(0)).max() / 2)
    one = torch.ones_like(X[:, :1])
    h = torch.cat([(X - mid) / s, one], 1)
    c0, w0, sp = meta['width'] / 2, meta['height'] / 2, max(meta['width'], meta['height']) / 2
    cn, wn, z = ((c - c0) / sp)[:, None], ((w - w0) / sp)[:, None], torch.zeros_like(h)
    A = torch.cat([torch.cat([h, z, -cn * h], 1), torch.cat([z, h, -wn * h], 1)])
    R = torch.linalg.qr(A, mode='r').R.cpu().numpy()
    T = np.eye(4) * s                                  # X = T h
    T[:3, 3], T[3, 3] = mid.cpu().numpy(), 1.0
    M = np.zeros((12, 12))                             # normalised rows from the camera's own
    M[0:4, 0:4] = M[4:8, 4:8] = T.T / sp
    M[0:4, 8:12], M[4:8, 8:12], M[8:12, 8:12] = -T.T * c0 / sp, -T.T * w0 / sp, T.T
    P = np.linalg.svd(R @ M)[2][11].reshape(3, 4)
    q, r = np.linalg.qr(P[::-1, :3].T)                 # RQ of the left block, positive diagonal
    sign = np.sign(np.diag(r))
    K, Q = (r * sign[:, None]).T[::-1, ::-1], (q * sign).T[::-1]
    P, K = P / K[2, 2], K / K[2, 2]
    if np.linalg.det(Q) < 0:
        Q, P = -Q, -P
    t = np.linalg.solve(K, P[:, 3])
    w4 = np.array([Q[0, 0] + Q[1, 1] + Q[2, 2], Q[0, 0] - Q[1, 1] - Q[2, 2], Q[1, 1] - Q[0, 0] - Q[2, 2],
                   Q[2, 2] - Q[0, 0] - Q[1, 1]])
    i = int(np.argmax(w4))
    f = 2.0 * math.sqrt(1.0 + w4[i])                   # four times the largest quaternion part
    a, b, e = Q[2, 1] - Q[1, 2], Q[0, 2] - Q[2, 0], Q[1, 0] - Q[0, 1]
    u, v, y = Q[0, 1] + Q[1, 0], Q[0, 2] + Q[2, 0], Q[1, 2] + Q[2, 1]
    quat = np.array([[f * f / 4, a, b, e], [a, f * f / 4, u, v], [b, u, f * f / 4, y], [e, v, y, f * f / 4]][i]) / f
    params = [meta['width'], meta['height'], K[0, 0], K[1, 1], K[0, 2], K[1, 2], K[0, 1], *quat, *t]
    Kd, Qd, td = (torch.tensor(np.ascontiguousarray(m), dtype=F64, device='cuda') for m in (K, Q, t))
    cam = X @ Qd.T + td
    p = cam @ Kd.T
    pe = torch.hypot(p[:, 0] / p[:, 2] - c, p[:, 1] / p[:, 2] - w)
    ray = torch.cat([c[:, None], w[:, None], one], 1) @ torch.linalg.inv(Kd).T
    ie = ((cam * ray).sum(1, keepdim=True) / (ray * ray).sum(1, keepdim=True) * ray - cam).norm(dim=1)
    mid2 = lambda d: (d.sort().values[(d.numel() - 1) // 2] + d.sort().values[d.numel() // 2]) / 2  # noqa: E731
    err = torch.stack([pe.mean(), mid2(pe), pe.max(), ie.mean(), mid2(ie), ie.max()])
    return torch.tensor(params, dtype=F64, device='cuda'), err


def _exact_affine(metas, g):
    rows = []
    for m in metas:
        col, row = _project(m, g['lat'], g['lon'], g['alt'])
        k = _inside(m, col, row)
        a = torch.stack([g['lat'][k], g['lon'][k], g['alt'][k]], 1)
        mid, half = (a.amax(0) + a.amin(0)) / 2, (a.amax(0) - a.amin(0)) / 2
        a = torch.cat([(a - mid) / half, torch.ones_like(a[:, :1])], 1)
        p = torch.linalg.solve(a.T @ a, a.T @ torch.stack([col[k], row[k]], 1)).T
        q = p[:, :3] / half
        rows.append(torch.cat([torch.tensor([m['width'], m['height']], dtype=F64, device='cuda'),
                               torch.cat([q, p[:, 3:] - (q * mid).sum(1, keepdim=True)], 1).reshape(-1)]))
    return torch.stack(rows), None


def _nanmax(points, xoff, yoff, res, xsize, ysize):
    row, col = torch.floor((yoff - points[:, 1]) / res), torch.floor((points[:, 0] - xoff) / res)
    ok = (row >= 0) & (col >= 0) & (row < ysize) & (col < xsize) & ~torch.isnan(points[:, 2])
    cell = (row[ok] * xsize + col[ok]).long()
    out = torch.full((ysize * xsize,), -math.inf, dtype=F64, device=points.device)
    out.scatter_reduce_(0, cell, points[ok, 2], 'amax')
    return torch.where(out == -math.inf, torch.full_like(out, math.nan), out).view(ysize, xsize)


def _shifts(pad):
    h, w = pad.shape[0] - 2, pad.shape[1] - 2
    return [pad[i:i + h, j:j + w] for i in range(3) for j in range(3)]


def _hole_fill(d):
    """NaN cells take the median of their valid 3x3 neighbours."""
    pad = torch.nn.functional.pad(d, (1, 1, 1, 1), value=math.nan)
    r, c = torch.nonzero(torch.isnan(d), as_tuple=True)
    if not r.numel():
        return d
    s = torch.sort(torch.stack([pad[r + i, c + j] for i in range(3) for j in range(3)], 1), dim=1).values
    n = (~torch.isnan(s)).sum(1)
    lo = s.gather(1, ((n - 1) // 2).clamp(min=0)[:, None])[:, 0]
    hi = s.gather(1, (n // 2).clamp(max=8)[:, None])[:, 0]
    out = d.clone()
    out[r, c] = (lo + hi) / 2
    return out


def _blur(d):
    """cv2.medianBlur(float32, 3): the 9-input network and its two compare-exchanges, which
    order NaN differently in the columns that run four at a time."""
    h, w = d.shape
    p = _shifts(torch.nn.functional.pad(d[None, None], (1, 1, 1, 1), mode='replicate')[0, 0])
    col = torch.arange(w, device=d.device)
    vec = (col >= 1) & (col < 1 + 4 * (((w - 6) // 4 + 1) if w >= 6 else 0))
    for a, b in ((1, 2), (4, 5), (7, 8), (0, 1), (3, 4), (6, 7), (1, 2), (4, 5), (7, 8), (0, 3), (5, 8), (4, 7), (3, 6),
                 (1, 4), (2, 5), (4, 7), (4, 2), (6, 4), (4, 2)):
        x = torch.where(vec, ~(p[a] < p[b]), p[b] < p[a])
        p[a], p[b] = torch.where(x, p[b], p[a]), torch.where(x, p[a], p[b])
    return p[4]


def _fuse(d):
    """(V, H, W) -> the mean of the heights within one MAD of their median, blurred."""
    v = d.shape[0]
    out = torch.empty(d.shape[1:], dtype=F64, device=d.device)

    def nanmedian(a, n):
        s = torch.sort(a, dim=0).values
        lo = s.gather(0, ((n - 1) // 2).clamp(min=0)[None])[0]
        return (lo + s.gather(0, (n // 2).clamp(max=v - 1)[None])[0]) / 2

    step = max(1, int(4e7 // (v * d.shape[2])))
    for r in range(0, d.shape[1], step):
        x = d[:, r:r + step].to(F64)
        n = (~torch.isnan(x)).sum(0)
        dev = (x - nanmedian(x, n)).abs()
        x = torch.where(dev > nanmedian(dev, n), torch.full_like(x, math.nan), x)
        out[r:r + step] = torch.where(n <= 2, torch.full_like(x[0], math.nan), x.nanmean(0))
    return _blur(out)


@functools.lru_cache(maxsize=None)
def _krueger():
    """Transverse Mercator from geodetic latitude (Karney 2011): Krueger's alpha to n^6."""
    f = 1.0 / 298.257223563
    n = f / (2.0 - f)
    alpha = (n / 2 - 2 * n**2 / 3 + 5 * n**3 / 16 + 41 * n**4 / 180 - 127 * n**5 / 288 + 7891 * n**6 / 37800,
             13 * n**2 / 48 - 3 * n**3 / 5 + 557 * n**4 / 1440 + 281 * n**5 / 630 - 1983433 * n**6 / 1935360,
             61 * n**3 / 240 - 103 * n**4 / 140 + 15061 * n**5 / 26880 + 167603 * n**6 / 181440,
             49561 * n**4 / 161280 - 179 * n**5 / 168 + 6601661 * n**6 / 7257600,
             34729 * n**5 / 80640 - 3418889 * n**6 / 1995840, 212378941 * n**6 / 319334400)
    return alpha, 6378137.0 / (1 + n) * (1 + n**2 / 4 + n**4 / 64 + n**6 / 256), f * (2.0 - f)


def _utm_points(depth, m, aoi, zone, south):
    """Depth map -> ENU -> geodetic (fixed-point iteration) -> UTM points."""
    alpha, rect, e2 = _krueger()
    a = 6378137.0
    h, w = depth.shape
    m = torch.tensor(np.asarray(m), dtype=F64, device='cuda')
    d = depth.to(F64)
    c = torch.arange(w, device='cuda', dtype=F64)[None, :]
    r = torch.arange(h, device='cuda', dtype=F64)[:, None]
    t = [m[i, 0] * c + m[i, 1] * r + m[i, 2] + m[i, 3] * d for i in range(4)]
    ok = depth > 0
    e, n, u = (t[i][ok] / t[3][ok] for i in range(3))
    lat0, lon0 = math.radians((aoi['lat_min'] + aoi['lat_max']) / 2), math.radians((aoi['lon_min'] + aoi['lon_max']) / 2)
    s0, c0, sl, cl = math.sin(lat0), math.cos(lat0), math.sin(lon0), math.cos(lon0)
    nu = a / math.sqrt(1 - e2 * s0 * s0)
    tt = c0 * u - s0 * n
    x = (nu + aoi['alt_min']) * c0 * cl + cl * tt - sl * e
    y = (nu + aoi['alt_min']) * c0 * sl + sl * tt + cl * e
    z = (nu * (1 - e2) + aoi['alt_min']) * s0 + s0 * u + c0 * n
    p = torch.hypot(x, y)
    lat = torch.atan2(z, p * (1 - e2))
    for _ in range(8):
        sn = torch.sin(lat)
        nn = a / torch.sqrt(1 - e2 * sn * sn)
        lat = torch.atan2(z + e2 * nn * sn, p)
    sn = torch.sin(lat)
    nn = a / torch.sqrt(1 - e2 * sn * sn)
    alt = p * torch.cos(lat) + z * sn - a * a / nn
    dl = torch.atan2(y, x) - math.radians((zone - 1) * 6 - 177)
    tau, ee = torch.tan(lat), math.sqrt(e2)
    sig = torch.sinh(ee * torch.atanh(ee * tau / torch.sqrt(1 + tau * tau)))
    tp = tau * torch.sqrt(1 + sig * sig) - sig * torch.sqrt(1 + tau * tau)
    xi, eta = torch.atan2(tp, torch.cos(dl)), torch.asinh(torch.sin(dl) / torch.sqrt(tp * tp + torch.cos(dl)**2))
    east, north = eta.clone(), xi.clone()
    for j, al in enumerate(alpha, 1):
        north += al * torch.sin(2 * j * xi) * torch.cosh(2 * j * eta)
        east += al * torch.cos(2 * j * xi) * torch.sinh(2 * j * eta)
    return torch.stack([500000.0 + 0.9996 * rect * east, 0.9996 * rect * north + (1e7 if south else 0.0), alt], 1)


def _map_points(m, aff):
    h, w = m.shape
    dj = 2 * torch.arange(w, device='cuda', dtype=F64)[None, :] + 1 - w
    di = 2 * torch.arange(h, device='cuda', dtype=F64)[:, None] + 1 - h
    e = (aff['e0'] + aff['ej'] * dj + aff['ei'] * di) * 2.0**-28
    n = (aff['n0'] + aff['nj'] * dj + aff['ni'] * di) * 2.0**-28
    return torch.stack([e.reshape(-1), n.reshape(-1), m.reshape(-1).to(F64)], 1)


def exact(case, seed):
    kind = case['kind']
    st = prepare(case, seed)
    if kind == 'project':
        ps = [_project(m, *st['points']) for m in st['metas']]
        if 'model' in st:
            return ps[0]
        out = (torch.stack([p[0] for p in ps]), torch.stack([p[1] for p in ps]))
        return out + (None,) if case['keep'] else out
    if kind == 'cube':
        x, y, z = st['xyz'].to(F64)
        out = torch.empty((case['cams'], 2, case['n']), dtype=F64, device='cuda')
        for k, m in enumerate(st['metas']):
            r = m['rpc']
            c, w = _rfm(r, x, y, z)
            out[k, 0], out[k, 1] = c * r['colScale'] + r['colOff'], w * r['rowScale'] + r['rowOff']
        return out
    if kind == 'inverse':
        return _exact_inverse(st['meta'], *st['points'])
    if kind == 'fit':
        fits = [_exact_fit(m, {k: t if case['shared'] else t[v] for k, t in st['grid'].items()})
                for v, m in enumerate(st['metas'])]
        return torch.stack([f[0] for f in fits]), torch.stack([f[1] for f in fits]), None
    if kind == 'affine':
        return _exact_affine(st['metas'], st['grid'])
    if kind == 'grid':
        d = _hole_fill(_nanmax(st['points'], synth.EXPLORER_UL_EASTING, synth.EXPLORER_UL_NORTHING, case['res'],
                               case['cells_x'], case['cells_y']))
        return d, _blur(d)
    if kind == 'dsm':
        o = st['offsets'].tolist()
        return torch.stack([_blur(_hole_fill(_nanmax(st['points'][a:b], synth.EXPLORER_UL_EASTING,
                                                     synth.EXPLORER_UL_NORTHING, case['res'], case['cells_x'],
                                                     case['cells_y']))) for a, b in zip(o, o[1:])])
    if kind == 'depth':
        xo, yo, res, _, xs, ys = st['grid']
        zone, south = st['aoi']['zone_number'], st['aoi']['hemisphere'] == 'S'
        return torch.stack([_blur(_hole_fill(_nanmax(_utm_points(d, m, st['aoi'], zone, south), xo, yo, res, xs, ys)))
                            for d, m in zip(st['depths'], st['mats'])])
    if kind == 'fuse':
        return _fuse(st['dsms'] if case['layout'] == 'vhw' else st['dsms'].permute(2, 0, 1))
    views, fused, k = [], [], 0
    for s, affs in zip(st['specs'], st['affines']):
        ds = []
        for a in affs:
            pts = _map_points(st['pool'][k % 6][:s.image, :s.image], a)
            ds.append(_blur(_hole_fill(_nanmax(pts, s.xoff, s.yoff, s.res, s.xsize, s.ysize))))
            k += 1
        views += [d.reshape(-1) for d in ds]
        fused.append(_fuse(torch.stack(ds).to(torch.float32)).reshape(-1))
    return torch.cat(fused), torch.cat(views)
