"""Exact RPC projection at the edges of its integer products: every result has the bits of
the FP64 restatement of lib/rpc_model.py:160-168 (tolerance: none)."""
import numpy as np
import pytest

from conftest import same_bits
from oracle import rpc as orpc

pytestmark = pytest.mark.gpu


def _camera(kind):
    from vissatsatellitestereo_gb300 import synth
    m = synth.make_rpc_meta(31, 4096, 3000)
    r = m['rpc']
    rng = np.random.default_rng(8)
    if kind == 'zeros':                # zero terms of either sign, zero constant terms
        for key in ('rowNum', 'rowDen', 'colNum', 'colDen'):
            c = np.array(r[key])
            c[rng.choice(np.arange(3, 20), 9, replace=False)] = 0.0
            c[19] = -0.0
            r[key] = c.tolist()
        r['colNum'][0] = 0.0
        r['rowNum'][0] = -0.0
    elif kind == 'dyadic':             # few significant bits: products that end in ties
        for key in ('rowNum', 'rowDen', 'colNum', 'colDen'):
            c = np.array(r[key])
            r[key] = (np.round(c * 2.0**30) * 2.0**-30 + 2.0**-52 * (c > 0)).tolist()
        r['latScale'], r['lonScale'], r['altScale'] = 2.0 - 2.0**-52, 1.0 / 3.0, 0.1
        r['latOff'], r['lonOff'], r['altOff'] = 0.0, 0.0, 0.0
    elif kind == 'wide':               # coefficients whose products leave the normal range
        r['colNum'][11] = 1e-300
        r['rowNum'][19] = 1e-60
        r['colDen'][15] = 1e150
    elif kind == 'scale':
        r['lonScale'] = 5e-320
    return m


def _points(kind, m, n):
    r = m['rpc']
    rng = np.random.default_rng(9)
    u = rng.uniform(-1.05, 1.05, (3, n))
    if kind == 'dyadic':
        u = np.round(u * 64) / 64
    lat, lon, alt = (r[k + 'Off'] + r[k + 'Scale'] * v for k, v in zip(('lat', 'lon', 'alt'), u))
    if kind == 'zero':                 # coordinates on their offsets, alone and together
        lat[::2], lon[::3], alt[::5] = r['latOff'], r['lonOff'], r['altOff']
    if kind == 'extreme':
        odd = np.array([np.inf, -np.inf, np.nan, 0.0, -0.0, 5e-324, 1e-310, 1e308, -1e200, 1e60, 1e-60])
        for k, a in enumerate((lat, lon, alt)):
            a[k::7] = odd[np.arange(a[k::7].size) % odd.size]
    return lat, lon, alt


@pytest.mark.parametrize('points', ['random', 'zero', 'dyadic', 'extreme'])
@pytest.mark.parametrize('cam', ['plain', 'zeros', 'dyadic', 'wide', 'scale'])
def test_exact_projection_has_the_reference_bits(cam, points):
    from vissatsatellitestereo_gb300.rpc_model import RPCModel
    m = _camera(cam)
    for n in (1, 31, 33, 5000):
        p = _points(points, m, n)
        with np.errstate(all='ignore'):
            want = orpc.projection(m, *p)
        got = RPCModel(m).projection(*p)
        assert same_bits(got[0], want[0]) and same_bits(got[1], want[1]), n


@pytest.mark.parametrize('n', [20000, 80000, 200001])
def test_exact_projection_over_the_block_sizes(n):
    """Launches of every block size, several cameras, masks."""
    from vissatsatellitestereo_gb300.rpc_model import project_cameras
    ms = [_camera(k) for k in ('plain', 'zeros')]
    p = _points('random', ms[0], n)
    col, row, keep = (t.cpu().numpy() for t in project_cameras(ms, *p, mode='exact', keep=True))
    for c, m in enumerate(ms):
        want = orpc.projection(m, *p)
        assert same_bits(col[c], want[0]) and same_bits(row[c], want[1])
        assert np.array_equal(keep[c] != 0, orpc.in_image(m, *want))


@pytest.mark.parametrize('cam', ['plain', 'zeros'])
@pytest.mark.parametrize('n', [1, 31, 64, 65, 4097])
def test_inverse_projection_has_the_reference_bits(cam, n):
    from vissatsatellitestereo_gb300.rpc_model import RPCModel
    m = _camera(cam)
    rng = np.random.default_rng(n)
    r = m['rpc']
    col, row = rng.uniform(0, m['width'], n), rng.uniform(0, m['height'], n)
    alt = r['altOff'] + r['altScale'] * rng.uniform(-0.5, 0.5, n)
    alt[::2] = r['altOff']
    model = RPCModel(m)
    lon, lat, _ = model.inverse_projection(col, row, alt)
    lo, la, _, its = orpc.inverse_projection(m, col, row, alt)
    assert same_bits(lon, lo) and same_bits(lat, la) and model.last_iterations == its


def test_inverse_projection_reports_a_point_that_never_converges():
    import torch
    from vissatsatellitestereo_gb300._lib import VS_ERR_DEGENERATE, VsError
    from vissatsatellitestereo_gb300.rpc_model import inverse_project_cameras
    ms = [_camera('plain'), _camera('zeros')]
    col = torch.full((40,), 700.0, dtype=torch.float64, device='cuda')
    bad = col.clone()
    bad[7] = float('nan')
    with pytest.raises(VsError) as e:
        inverse_project_cameras(ms, bad, col, col, max_iter=12)
    assert e.value.status == VS_ERR_DEGENERATE
    with pytest.raises(VsError):
        inverse_project_cameras(ms, col, col, col, max_iter=1)
