"""Fusion of more than 64 views at the shares where the network of a lane changes (44 and 52 values), for 2, 4 and
8 lanes per cell, against the oracle restatement of aggregate_2p5d.py:65-81 (bit-exact)."""
import numpy as np
import pytest

from conftest import same_bits
from oracle import fuse

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('layout', ['hwv', 'vhw'])
@pytest.mark.parametrize('V', [88, 89, 104, 105, 176, 177, 208, 209, 352, 353, 416, 417])
def test_fusion_where_the_network_changes(V, layout):
    import torch
    from vissatsatellitestereo_gb300.aggregate_2p5d import fuse_dsms
    rng = np.random.default_rng(V)
    d = (rng.normal(30.0, 10.0, (9, 13, 1)) + rng.normal(0.0, 0.5, (9, 13, V))).astype(np.float32)
    d[1:][rng.random((8, 13, V)) < 0.15] = np.nan         # the first row keeps all of its views
    with np.errstate(all='ignore'):
        want = fuse.fuse_numpy(d)
    src = torch.from_numpy(d if layout == 'hwv' else np.ascontiguousarray(d.transpose(2, 0, 1))).cuda()
    assert same_bits(fuse_dsms(src, median_blur=False, layout=layout).cpu().numpy(), want)
