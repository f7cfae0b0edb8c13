"""Fusion of more than 64 views (several lanes per cell) at the edges of its shares, tiles and
layouts, against the oracle restatement of aggregate_2p5d.py:65-81 (bit-exact)."""
import numpy as np
import pytest

from conftest import same_bits
from oracle import blur, fuse

pytestmark = pytest.mark.gpu


def _stack(V, h, w, odd):
    rng = np.random.default_rng(V * 100 + h)
    d = (rng.normal(30.0, 10.0, (h, w, 1)) + rng.normal(0.0, 0.5, (h, w, V))).astype(np.float32)
    d[rng.random((h, w, V)) < 0.15] = np.nan
    d[0, 0] = np.nan                                     # cells of 0, 2 and 3 valid views
    d[0, 1, 2:] = np.nan
    d[0, 2, 3:] = np.nan
    d[1, 0] = np.where(np.arange(V) % 2, np.float32(0.0), np.float32(-0.0))
    d[1, 1] = np.float32(7.25)                            # all equal
    if odd:                                              # infinite medians, one infinity, all of one sign
        d[2, 0, :] = np.inf
        d[2, 1, : V // 2 + 5] = np.inf
        d[2, 2, :3] = -np.inf
        d[2, 3, : V // 2], d[2, 3, V // 2:] = -np.inf, np.inf
    return d


@pytest.mark.parametrize('layout', ['hwv', 'vhw'])
@pytest.mark.parametrize('V', [65, 95, 96, 97, 127, 128, 129, 191, 193, 255, 256, 257, 385, 511, 512])
def test_wide_fusion_matches_oracle(V, layout):
    import torch
    from vissatsatellitestereo_gb300.aggregate_2p5d import fuse_dsms
    for h, w, odd in ((7, 9, True), (8, 36, False)):
        d = _stack(V, h, w, odd)
        with np.errstate(all='ignore'):
            want = fuse.fuse_numpy(d)
        src = torch.from_numpy(d if layout == 'hwv' else np.ascontiguousarray(d.transpose(2, 0, 1))).cuda()
        got = fuse_dsms(src, median_blur=False, layout=layout).cpu().numpy()
        assert same_bits(got, want)
        blurred = fuse_dsms(src, median_blur=True, layout=layout).cpu().numpy()
        assert same_bits(blurred, blur.median_blur3x3(want))
