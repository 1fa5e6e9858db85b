"""Workspace sizes of sdp_hogbom: the deferred-update kernel's tables come on
top of what the other kernels need (the size asked for grids above 16383,
where that kernel never runs).  A workspace of the smaller size serves every
grid, with the oracle's results bit for bit; one byte less is refused.  So does
one on any 8-byte boundary, which the deferred kernel's 16-byte entries could
not use."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(G):
    rng = np.random.default_rng(G)
    yy, xx = np.mgrid[0:G, 0:G]
    psf = np.exp(-((xx - G // 2) ** 2 + (yy - G // 2) ** 2) / 8.0).astype(np.float32).reshape(-1)
    res = (0.01 * rng.standard_normal(G * G)).astype(np.float32)
    res[rng.integers(0, G * G, 12)] += 1.0
    return res, psf


def _check(device, params, psf_d, res, ref, workspace):
    import torch
    n1, s1, m1, r1 = ref
    G, minor = params.grid_size, params.num_minor_cycles
    r, m = torch.from_numpy(res.copy()).cuda(), torch.zeros(G * G, device="cuda")
    s, c = torch.zeros((minor, 3), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    device.hogbom(params, r, psf_d, m, s, c, workspace)
    assert int(c.item()) == n1
    np.testing.assert_array_equal(s[:n1].cpu().numpy(), s1)
    np.testing.assert_array_equal(m.cpu().numpy(), m1)
    np.testing.assert_array_equal(r.cpu().numpy(), r1)


@pytest.mark.parametrize("G", [256, 2784])
def test_smaller_workspace(sdp, device, oracle32, G):
    import torch
    minor = 20
    small, full = device.hogbom_workspace_bytes(16384), device.hogbom_workspace_bytes(G)
    assert small < full
    res, psf = _scene(G)
    ref = oracle32.hogbom(G, minor, minor, res, psf, 1.0, 1e-5)
    params = sdp.CleanParams(G, minor, minor, 0.1, 1.5, 0.0002, 1.0, 1e-5)
    p = torch.from_numpy(psf).cuda()
    for size in (small, full):
        guard = torch.full((size + 4096,), 0x5a, dtype=torch.uint8, device="cuda")
        _check(device, params, p, res, ref, guard[:size])
        assert bool((guard[size:] == 0x5a).all())
    with pytest.raises(sdp.SdpError, match="workspace"):
        _check(device, params, p, res, ref, guard[:small - 1])


def test_workspace_on_an_8_byte_boundary(sdp, device, oracle32):
    import torch
    G, minor = 2784, 20
    size = device.hogbom_workspace_bytes(G)
    res, psf = _scene(G)
    ref = oracle32.hogbom(G, minor, minor, res, psf, 1.0, 1e-5)
    params = sdp.CleanParams(G, minor, minor, 0.1, 1.5, 0.0002, 1.0, 1e-5)
    guard = torch.empty(size + 256, dtype=torch.uint8, device="cuda")
    assert guard.data_ptr() % 16 == 0
    _check(device, params, torch.from_numpy(psf).cuda(), res, ref, guard[8:8 + size])
