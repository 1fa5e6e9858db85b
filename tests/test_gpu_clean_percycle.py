"""Hogbom with one launch per minor cycle (k_clean_cycle): images that do not
fit on chip where the noise test could stop the loop (noise factor x gain >=
0.5, so every minor cycle needs the mean of |r|).  Components, model and
residual against the oracle bit for bit, with a noise test that never fires
and with one that ends the loop, for sides with and without four-pixel
chunks."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_clean_deferred import _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G,noise,stops", [(2816, 5.1, False), (2816, 250.0, True), (2755, 5.1, False), (2755, 250.0, True)])
def test_against_the_oracle(sdp, device, oracle32, G, noise, stops):
    import torch
    minor = 200
    res, psf = _scene(G, 8, 0.01, 2e-3, G)
    n1, s1, m1, r1 = oracle32.hogbom(G, minor, minor, res, psf, 3.0, 1e-5, noise_factor=noise)
    assert (10 < n1 < minor) if stops else n1 == minor
    params = sdp.CleanParams(G, minor, minor, 0.1, noise, 0.0002, 3.0, 1e-5)
    r, p = torch.from_numpy(res.copy()).cuda(), torch.from_numpy(psf).cuda()
    m, s = torch.zeros(G * G, device="cuda"), torch.zeros((minor, 3), device="cuda")
    c = torch.zeros(1, dtype=torch.int32, device="cuda")
    ws = torch.empty(device.hogbom_workspace_bytes(G), dtype=torch.uint8, device="cuda")
    device.hogbom(params, r, p, m, s, c, ws)
    assert int(c.item()) == n1
    np.testing.assert_array_equal(s[:n1].cpu().numpy(), s1)
    np.testing.assert_array_equal(m.cpu().numpy(), m1)
    np.testing.assert_array_equal(r.cpu().numpy(), r1)
