"""Perspective fit at the edges of a moment block's span of 2048 points, in a form that sees every point: one
observation at an edge of the span is far off, and the camera moves as the oracle's does.  Bar: 1e-3 px of
reprojection (as for the full-size fits); the far point moves the oracle's camera by more than ten times
that."""
import numpy as np
import pytest

from oracle import dlt, rpc

pytestmark = pytest.mark.gpu
PX_TOL = 1e-3


def _points(n):
    from vissatsatellitestereo_gb300 import synth
    meta = synth.make_rpc_meta(77, 4096, 4096)
    g = synth.rpc_sample_grid(meta, 24, 10)
    col, row = rpc.projection(meta, g.lat, g.lon, g.alt)
    pick = np.flatnonzero(rpc.in_image(meta, col, row).ravel())
    pick = np.random.default_rng(n).permutation(pick)
    pick = np.resize(pick, n)
    return meta, {k: np.ascontiguousarray(v.ravel()[pick]) for k, v in
                  dict(x=g.x, y=g.y, z=g.z, lat=g.lat, lon=g.lon, alt=g.alt, col=col, row=row).items()}


def _moves(a, b, p):
    c0, r0 = dlt.reproject(*a, p['x'], p['y'], p['z'])
    c1, r1 = dlt.reproject(*b, p['x'], p['y'], p['z'])
    return np.max(np.hypot(c1 - c0, r1 - r0))


def _edges(n):
    return sorted({k for k in (0, 127, 128, 255, 2046, 2047, 2048, 4095, 4096, n - 2, n - 1) if 0 <= k < n})


@pytest.mark.parametrize('n', [255, 2047, 2048, 2049, 2050, 4096, 4097])
def test_fit_sees_the_points_at_the_edges(n):
    from vissatsatellitestereo_gb300.solve_perspective import solve_perspective_batch
    _, p = _points(n)
    keep = np.ones(n, bool)
    keep[1::7] = False
    clean = dlt.solve_perspective(p['x'], p['y'], p['z'], p['col'], p['row'], keep)
    edges = [e for e in _edges(n) if keep[e]]
    cols = np.repeat(p['col'][None], len(edges), 0)
    cols[np.arange(len(edges)), edges] += 0.4 * n              # one view per far observation
    rows = np.repeat(p['row'][None], len(edges), 0)
    got = [o.cpu().numpy() for o in solve_perspective_batch(p['x'], p['y'], p['z'], cols, rows,
                                                            np.repeat(keep[None], len(edges), 0))]
    for v, e in enumerate(edges):
        want = dlt.solve_perspective(p['x'], p['y'], p['z'], cols[v], rows[v], keep)
        assert _moves(clean, want, p) > 10 * PX_TOL, e
        assert got[3][v] == 0 and _moves([g[v] for g in got[:3]], want, p) < PX_TOL, e


@pytest.mark.parametrize('n', [2047, 2048, 2049, 4097])
def test_camera_fit_sees_the_points_at_the_edges(n):
    from vissatsatellitestereo_gb300.camera_approx import approx_perspective_enu, params_to_krt
    meta, p = _points(n)
    clean = dlt.solve_perspective(p['x'], p['y'], p['z'], p['col'], p['row'])
    edges = _edges(n)
    per_view = {k: np.repeat(p[k][None], len(edges), 0) for k in ('lat', 'lon', 'alt', 'x', 'y', 'z')}
    per_view['x'][np.arange(len(edges)), edges] += 0.2 * n     # metres
    params, _, status = approx_perspective_enu([meta] * len(edges), *per_view.values(), mode='exact', shared_points=False)
    assert not status.any()
    for v, e in enumerate(edges):
        x = per_view['x'][v]
        want = dlt.solve_perspective(x, p['y'], p['z'], p['col'], p['row'])
        assert _moves(clean, want, p) > 10 * PX_TOL, e
        assert _moves(params_to_krt(params[v].cpu().numpy()), want, p) < PX_TOL, e
