"""Perspective fit and error statistics at the edges of their reductions: few points, no kept
points, ties, views of different fate in one call.  Bar of the statistics: 1e-3 px / m (as for
the full-size fits); a view in a batch has the bits of the view alone."""
import numpy as np
import pytest

from conftest import same_bits
from oracle import dlt, rpc

pytestmark = pytest.mark.gpu


def _problem(n, seed):
    from vissatsatellitestereo_gb300 import synth
    meta = synth.make_rpc_meta(400 + seed, 4096, 4096)
    g = synth.rpc_sample_grid(meta, 24, 10)
    rng = np.random.default_rng(seed)
    pick = rng.permutation(g.n)[:n] if n <= g.n else rng.integers(0, g.n, n)
    col, row = rpc.projection(meta, g.lat, g.lon, g.alt)
    x, y, z, c, r = (a.ravel()[pick] for a in (g.x, g.y, g.z, col, row))
    full = dlt.solve_perspective(*(a.ravel() for a in (g.x, g.y, g.z, col, row)))
    return x, y, z, c, r, full


@pytest.mark.parametrize('n', [1, 2, 3, 31, 255, 257, 1024, 5001])
def test_error_statistics_of_few_points(n):
    from vissatsatellitestereo_gb300.check_error import perspective_error_batch
    x, y, z, c, r, (K, R, t) = _problem(n, n)
    keep = np.ones(n, bool)
    keep[1::3] = False
    got = perspective_error_batch(x, y, z, c[None], r[None], K[None], R[None], t[None], keep[None]).cpu().numpy()[0]
    want = dlt.perspective_error(*(a.reshape(-1, 1) for a in (x, y, z, c, r)), K, R, t, keep)
    assert np.max(np.abs(got - want)) < 1e-3


def test_statistics_of_equal_errors_and_of_no_points():
    from vissatsatellitestereo_gb300.check_error import perspective_error_batch
    x, y, z, c, r, (K, R, t) = _problem(1, 5)
    rep = lambda a: np.repeat(a, 999)  # noqa: E731
    one = perspective_error_batch(x, y, z, c[None], r[None], K[None], R[None], t[None]).cpu().numpy()[0]
    many = perspective_error_batch(rep(x), rep(y), rep(z), rep(c)[None], rep(r)[None], K[None], R[None],
                                   t[None]).cpu().numpy()[0]
    assert np.array_equal(many[[1, 2, 4, 5]], one[[1, 2, 4, 5]]) and np.allclose(many, one, rtol=1e-6)
    none = perspective_error_batch(x, y, z, c[None], r[None], K[None], R[None], t[None],
                                   np.zeros((1, 1), bool)).cpu().numpy()[0]
    assert np.all(np.isnan(none))


@pytest.mark.parametrize('n', [5, 6, 7, 240, 5001])
def test_views_in_a_batch_equal_views_alone(n):
    """A good view, one with too few kept points, one whose points lie in a plane."""
    from vissatsatellitestereo_gb300._lib import VS_ERR_DEGENERATE
    from vissatsatellitestereo_gb300.solve_perspective import solve_perspective_batch
    ps = [_problem(n, s) for s in (1, 2, 3)]
    x, y, z, c, r = (np.stack([p[k] for p in ps]) for k in range(5))
    z[2] = 0.0
    keep = np.ones((3, n), bool)
    keep[1, 5:] = False
    both = [a.cpu().numpy() for a in solve_perspective_batch(x, y, z, c, r, keep, shared_points=False)]
    for v in range(3):
        alone = [a.cpu().numpy() for a in solve_perspective_batch(x[v], y[v], z[v], c[v:v + 1], r[v:v + 1], keep[v:v + 1])]
        assert int(both[3][v]) == int(alone[3][0])
        for b, a in zip(both[:3], alone[:3]):
            assert same_bits(b[v], a[0])
    assert int(both[3][1]) == VS_ERR_DEGENERATE and not both[0][1].any()
