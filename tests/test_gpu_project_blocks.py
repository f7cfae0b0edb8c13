"""Projection at the point counts where the block size changes (128 and 512 points per SM, in all cameras
together): a point's result does not depend on how many there are, and is the oracle's (exact form: the
same bits; fast form: 1e-4 px, its stated accuracy over the frame of the camera, here the first one's)."""
import numpy as np
import pytest
import torch

from conftest import same_bits
from oracle import rpc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('mode', ['exact', 'fast'])
@pytest.mark.parametrize('cams', [1, 3])
def test_results_do_not_depend_on_the_block_size(mode, cams):
    from vissatsatellitestereo_gb300 import synth
    from vissatsatellitestereo_gb300.rpc_model import project_cameras
    metas = [synth.make_rpc_meta(300 + k, 4096, 4096) for k in range(cams)]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    r = metas[0]['rpc']
    u = np.random.default_rng(1).uniform(-1.0, 1.0, (3, 600 * sms))
    pts = [torch.from_numpy(r[k + 'Off'] + r[k + 'Scale'] * v).cuda() for k, v in zip(('lat', 'lon', 'alt'), u)]
    whole = project_cameras(metas, *pts, mode=mode)
    host = [p[:2000].cpu().numpy() for p in pts]
    for c, m in enumerate(metas):
        for got, want in zip(whole, rpc.projection(m, *host)):
            got = got[c, :2000].cpu().numpy()
            if mode == 'exact':
                assert same_bits(got, want)
            elif c == 0:                       # the points lie far outside the other cameras' frames
                assert np.abs(got - want).max() < 1e-4
    for per_sm in (128, 512):
        edge = per_sm * sms // cams
        for n in (1, 255, 257, edge - 1, edge, edge + 1):
            part = project_cameras(metas, *(p[:n] for p in pts), mode=mode)
            for a, b in zip(part, whole):
                assert same_bits(a.cpu().numpy(), b[:, :n].cpu().numpy())
