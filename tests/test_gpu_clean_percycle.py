"""Hogbom with one launch per minor cycle (k_clean_cycle): images that do not
fit on chip where the noise test could stop the loop (noise factor x gain >=
0.5, so every minor cycle needs the mean of |r|).  Components, model and
residual against the oracle bit for bit, with a noise test that never fires
and with one that ends the loop, for sides with and without four-pixel
chunks."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(G):
    """Eight peaks of 1 on noise of 0.01, a PSF of one pixel with sidelobes everywhere."""
    rng = np.random.default_rng(G)
    psf = (1e-4 * rng.standard_normal((G, G))).astype(np.float32)
    psf[G // 2, G - G // 2] = 1.0  # the mirrored centre
    res = (0.01 * rng.standard_normal((G, G))).astype(np.float32)
    for y, x in rng.integers(0, G, (8, 2)):
        res[y, x] = 1.0
    return res.reshape(-1), psf.reshape(-1)


# gain 0.5: the peaks go down by halves, and the mean of |r| is 0.008, so a
# factor of 42 stops the loop between 0.25 and 0.125 (the oracle's running
# mean in floats is off by some 0.2 %)
@pytest.mark.parametrize("G", [2816, 2755])
@pytest.mark.parametrize("noise,minor,stops", [(1.1, 60, False), (42.0, 200, True)])
def test_against_the_oracle(sdp, device, oracle32, G, noise, minor, stops):
    import torch
    res, psf = _scene(G)
    n1, s1, m1, r1 = oracle32.hogbom(G, minor, minor, res, psf, 3.0, 1e-5, loop_gain=0.5, noise_factor=noise)
    assert n1 == (24 if stops else minor)
    params = sdp.CleanParams(G, minor, minor, 0.5, noise, 0.0002, 3.0, 1e-5)
    r, p = torch.from_numpy(res.copy()).cuda(), torch.from_numpy(psf).cuda()
    m, s = torch.zeros(G * G, device="cuda"), torch.zeros((minor, 3), device="cuda")
    c = torch.zeros(1, dtype=torch.int32, device="cuda")
    ws = torch.empty(device.hogbom_workspace_bytes(G), dtype=torch.uint8, device="cuda")
    device.hogbom(params, r, p, m, s, c, ws)
    assert int(c.item()) == n1
    np.testing.assert_array_equal(s[:n1].cpu().numpy(), s1)
    np.testing.assert_array_equal(m.cpu().numpy(), m1)
    np.testing.assert_array_equal(r.cpu().numpy(), r1)
