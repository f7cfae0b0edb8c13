"""Perspective fit at the edges of a moment block's span of points (2048), from arrays that start on
and off a 16-byte boundary: where the arrays start changes no bit."""
import numpy as np
import pytest
import torch

from conftest import same_bits
from oracle import rpc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n', [12, 256, 2047, 2048, 2049, 2050, 4097])
def test_fit_does_not_depend_on_where_the_arrays_start(n):
    from vissatsatellitestereo_gb300 import synth
    from vissatsatellitestereo_gb300.solve_perspective import solve_perspective_batch
    meta = synth.make_rpc_meta(77, 4096, 4096)
    g = synth.rpc_sample_grid(meta, 24, 10)
    pick = np.random.default_rng(n).permutation(g.n)[:n]
    col, row = rpc.projection(meta, g.lat, g.lon, g.alt)
    arrays = [np.ascontiguousarray(a.ravel()[pick]) for a in (g.x, g.y, g.z, col, row)]

    def fit(shift):
        dev = []
        for a in arrays:
            buf = torch.full((len(a) + shift,), float('nan'), dtype=torch.float64, device='cuda')
            buf[shift:] = torch.as_tensor(a, device='cuda')
            dev.append(buf[shift:])
        x, y, z, c, r = dev
        keep = torch.ones(1, len(x), dtype=torch.bool, device='cuda')
        keep[0, 1::5] = False
        return [o.cpu().numpy() for o in solve_perspective_batch(x, y, z, c[None], r[None], keep)]

    aligned, shifted = fit(0), fit(1)
    assert int(aligned[3][0]) == 0
    for a, b in zip(aligned, shifted):
        assert same_bits(a, b)
