"""Inverse projection where the points' iteration counts drift apart: points that leave the bound
again at the common count, counts past one launch's share, and calls that fail."""
import numpy as np
import pytest
import torch

from conftest import same_bits
from oracle import rpc as orpc

pytestmark = pytest.mark.gpu


def _camera(col):
    """A camera whose normalised frame is the raw one: column = the polynomial, row = latitude."""
    one, lat, num = np.zeros(20), np.zeros(20), np.zeros(20)
    one[0], lat[2] = 1.0, 1.0
    for k, c in col.items():
        num[k] = c
    r = {k + s: v for k in ('row', 'col', 'lat', 'lon', 'alt') for s, v in (('Off', 0.0), ('Scale', 1.0))}
    r.update(rowNum=lat.tolist(), rowDen=one.tolist(), colNum=num.tolist(), colDen=one.tolist())
    return {'rpc': r, 'width': 8, 'height': 8}


def leaving():
    """Column lon^2 + 5e-10 lon.  From lon = -1 the first difference is 1e-9, so a point within 5e-10 of
    its target (converged) is thrown to lon = 0 by the next iteration and comes back to it
    much later; a point with another row converges after one iteration."""
    m = _camera({7: 1.0, 1: 5e-10})
    n = 70
    col, row = np.full(n, 1.0 - 5e-10), np.linspace(-0.9, 0.9, n)
    col[37], row[37] = 1.0, -1.0
    return m, col, row, np.zeros(n)


def slow():
    """Column lon^3 + 0.0015 lon near its flat middle: linear convergence, some eighty iterations."""
    m = _camera({11: 1.0, 1: 0.0015})
    rng = np.random.default_rng(5)
    n = 130
    return m, rng.uniform(1e-7, 1e-3, n), rng.uniform(-0.5, 0.5, n), np.zeros(n)


def test_points_that_leave_the_bound_again():
    from vissatsatellitestereo_gb300 import synth
    from vissatsatellitestereo_gb300.rpc_model import inverse_project_cameras
    m, col, row, alt = leaving()
    lo, la, _, it = orpc.inverse_projection(m, col, row, alt)
    assert it > 4                                     # the first common count is 1
    plain = synth.make_rpc_meta(900, 2048, 2048)
    rng = np.random.default_rng(2)
    c2, r2 = rng.uniform(0, 2048, (2, len(col)))
    a2 = plain['rpc']['altOff'] + 0.0 * c2
    lo2, la2, _, it2 = orpc.inverse_projection(plain, c2, r2, a2)
    cams, sets = [plain, m, plain], [(c2, r2, a2), (col, row, alt), (c2, r2, a2)]
    lon, lat, _, its = inverse_project_cameras(cams, *(np.stack([s[k] for s in sets]) for k in range(3)), shared=False)
    assert its == [it2, it, it2]
    for c, (o, a) in enumerate([(lo2, la2), (lo, la), (lo2, la2)]):
        assert same_bits(lon[c].cpu().numpy(), o) and same_bits(lat[c].cpu().numpy(), a)


def test_counts_past_one_launch():
    from vissatsatellitestereo_gb300.rpc_model import inverse_project_cameras
    m, col, row, alt = slow()
    lo, la, _, it = orpc.inverse_projection(m, col, row, alt)
    assert it > 64
    m2, col2, row2, alt2 = leaving()
    lo2, la2, _, it2 = orpc.inverse_projection(m2, col2[:40], row2[:40], alt2[:40])
    n = len(col)
    fill = lambda v: np.resize(v[:40], n)
    lon, lat, _, its = inverse_project_cameras([m2, m], np.stack([fill(col2), col]), np.stack([fill(row2), row]),
                                               np.stack([fill(alt2), alt]), shared=False)
    assert its == [it2, it]
    assert same_bits(lon[1].cpu().numpy(), lo) and same_bits(lat[1].cpu().numpy(), la)
    assert same_bits(lon[0].cpu().numpy(), np.resize(lo2, n)) and same_bits(lat[0].cpu().numpy(), np.resize(la2, n))


@pytest.mark.parametrize('case', ['never', 'bound', 'leaves'])
def test_failed_call_leaves_its_outputs(case):
    """No camera's output is touched when one fails: a point that never converges, a bound below the
    count, a point that is converged once but not at the common count."""
    from vissatsatellitestereo_gb300 import _lib
    from vissatsatellitestereo_gb300._dev import ptr, stream_handle, workspace
    m, col, row, alt = leaving() if case == 'leaves' else slow()
    easy = _camera({1: 1.0})
    col, row, alt = (np.stack([np.zeros_like(v), v]) for v in (col, row, alt))
    if case == 'never':
        col[1, 3] = np.nan
    max_iter = {'never': 150, 'bound': 40, 'leaves': 3}[case]
    cams = torch.from_numpy(_lib.camera_array([easy, m])).cuda()
    n = col.shape[1]
    dev = [torch.from_numpy(v).cuda() for v in (col, row, alt)]
    out = [torch.full((2, n), 7.5, dtype=torch.float64, device='cuda') for _ in range(3)]
    wp, wb = workspace(_lib.lib().vs_rpc_inverse_project_workspace_size(2, n))
    with pytest.raises(_lib.VsError) as e:
        _lib.call('vs_rpc_inverse_project', ptr(cams), 2, *(ptr(d) for d in dev), n, n, 0, *(ptr(o) for o in out), max_iter,
                  None, wp, wb, stream_handle())
    assert e.value.status == _lib.VS_ERR_DEGENERATE and 'camera 1 ' in str(e.value)
    torch.cuda.synchronize()
    assert all(bool((o == 7.5).all()) for o in out)
