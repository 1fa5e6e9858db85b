"""Deferred CLEAN where the PSF map's blocks are larger than a tile (64 pixels
from a side of 4128 on): the bounds' indexing differs there.  A PSF with
sidelobes everywhere and components up to the corners, so that a bound that
missed a block would pass over a maximum; components, model and residual
against the oracle bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_clean_deferred import _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G,sidelobes", [(4161, 0.05), (4224, 0.2)])
def test_larger_blocks(sdp, device, oracle32, G, sidelobes):
    import torch
    minor = 50
    res, psf = _scene(G, 8, 0.01, sidelobes, G)
    n1, s1, m1, r1 = oracle32.hogbom(G, minor, minor, res, psf, 3.0, 1e-5)
    params = sdp.CleanParams(G, minor, minor, 0.1, 1.5, 0.0002, 3.0, 1e-5)
    r, p = torch.from_numpy(res.copy()).cuda(), torch.from_numpy(psf).cuda()
    m, s = torch.zeros(G * G, device="cuda"), torch.zeros((minor, 3), device="cuda")
    c = torch.zeros(1, dtype=torch.int32, device="cuda")
    ws = torch.empty(device.hogbom_workspace_bytes(G), dtype=torch.uint8, device="cuda")
    device.hogbom(params, r, p, m, s, c, ws)
    assert int(c.item()) == n1 == minor
    np.testing.assert_array_equal(s.cpu().numpy(), s1)
    np.testing.assert_array_equal(m.cpu().numpy(), m1)
    np.testing.assert_array_equal(r.cpu().numpy(), r1)
