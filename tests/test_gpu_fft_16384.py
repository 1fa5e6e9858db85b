"""The largest transform: columns of 16384 points over a cluster of eight CTAs
(2048-point parts of four columns), rows of 1024 threads, and a half spectrum
whose 8193 columns are no multiple of four.  Inputs whose transforms are known
in closed form, so that no second transform of that size is needed: a few
points (every column is dense in the second pass) and a few plane waves (every
row is dense in the first).  Bound as in test_gpu_fft_sizes."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

G = 16384
BOUND = 4 * 2.0 ** -24 * math.sqrt(2 * 14)
ROWS = 1024  # rows of a comparison at a time


def _wave(idx, k, sign):
    """exp(sign 2 pi i idx k / G) in doubles, the phase reduced in integers."""
    import torch
    t = ((idx * k) % G).double() * (2.0 * math.pi / G)
    return torch.complex(torch.cos(t), sign * torch.sin(t))


def _waves(parts, rows, sign):
    """Rows `rows` of the sum of a exp(sign 2 pi i (y r + x c) / G) over parts (y, x, a)."""
    import torch
    cols = torch.arange(G, device="cuda")
    out = 0
    for y, x, a in parts:
        out = out + a * _wave(rows, y, sign)[:, None] * _wave(cols, x, sign)[None, :]
    return out


def _error(got_rows, ref_rows):
    num = den = 0.0
    import torch
    for r0 in range(0, G, ROWS):
        rows = torch.arange(r0, r0 + ROWS, device="cuda")
        ref = ref_rows(rows)
        num += float((got_rows(rows) - ref).abs().square().sum())
        den += float(ref.abs().square().sum())
    return math.sqrt(num / den)


def _parts(seed):
    rng = np.random.default_rng(seed)
    p = [(int(y), int(x), complex(*rng.standard_normal(2))) for y, x in rng.integers(0, G, (3, 2))]
    return p + [(0, G - 1, 1.0 + 0.5j), (G // 2, 3, -0.7 + 0.2j)]


def _fill(parts, sign):
    import torch
    a = torch.empty((G, G, 2), device="cuda")
    for r0 in range(0, G, ROWS):
        rows = torch.arange(r0, r0 + ROWS, device="cuda")
        a[r0:r0 + ROWS] = torch.view_as_real(_waves(parts, rows, sign)).float()
    return a


def _points(parts):
    import torch
    a = torch.zeros((G, G, 2), device="cuda")
    for y, x, v in parts:
        a[y, x, 0] += v.real
        a[y, x, 1] += v.imag
    return a


@pytest.mark.parametrize("sign", [-1, 1])
def test_plain(sdp, device, sign):
    import torch
    parts = _parts(3)
    a, out = _points(parts), torch.empty((G, G, 2), device="cuda")
    device.fft2d(G, a, out, sign)
    assert _error(lambda r: torch.view_as_complex(out[r].double()), lambda r: _waves(parts, r, sign)) <= BOUND
    a = _fill(parts, -sign)
    device.fft2d(G, a, a, sign)  # in place
    ref = _points(parts).double()
    assert _error(lambda r: a[r].double() / G ** 2, lambda r: ref[r]) <= BOUND


def _sign(rows):
    import torch
    k = torch.arange(G, device="cuda")
    return 1.0 - 2.0 * ((rows[:, None] + k[None, :]) % 2).double()


def test_imaging_transforms(sdp, device):
    """image -> grid is C F(C image), grid -> image Re C F^-1(C grid) / taper, C the checkerboard."""
    import torch
    parts = _parts(4)
    work, out = (torch.empty((G, G, 2), device="cuda") for _ in range(2))
    real = [(y, x, complex(v.real)) for y, x, v in parts]
    image = _points(real)[..., 0].contiguous()
    device.image_to_grid(G, image, work, out)
    flip = [(y, x, v * (-1) ** ((y + x) % 2)) for y, x, v in real]
    assert _error(lambda r: torch.view_as_complex(out[r].double()), lambda r: _waves(flip, r, -1) * _sign(r)) <= BOUND
    # real plane waves: 2 Re (a wave) has its spectrum at (y, x) and the mirrored cell,
    # half the grid further on by the checkerboard
    for r0 in range(0, G, ROWS):
        rows = torch.arange(r0, r0 + ROWS, device="cuda")
        image[r0:r0 + ROWS] = (2.0 * _waves(parts, rows, 1).real).float()
    device.image_to_grid(G, image, work, out)
    ref = torch.zeros((G, G, 2), dtype=torch.float64, device="cuda")
    for y, x, v in parts:
        for yy, xx, w in ((y, x, v), (-y, -x, v.conjugate())):
            cy, cx = (yy + G // 2) % G, (xx + G // 2) % G
            s = (-1) ** ((cy + cx) % 2)
            ref[cy, cx, 0] += s * w.real
            ref[cy, cx, 1] += s * w.imag
    assert _error(lambda r: out[r].double() / G ** 2, lambda r: ref[r]) <= BOUND
    del ref
    prol = torch.empty(G // 2 + 1, device="cuda")
    device.prolate_table(G, prol)
    d = (torch.arange(G, device="cuda") - G // 2).abs()

    def keep(r):
        t = prol[d[r]][:, None] * prol[d][None, :]
        return t, (t.double().abs() > 1e-10) & (d[r] != 1229)[:, None] & (d != 1229)[None, :]

    def tapered(r):
        t, k = keep(r)
        assert not bool(image[r][~k].any())
        return torch.where(k, image[r].double() * t.double(), torch.zeros_like(t, dtype=torch.float64))

    def masked(r, x):
        return torch.where(keep(r)[1], x, torch.zeros_like(x))

    grid = _points(parts)
    device.grid_to_image(G, grid, prol, work, image)
    flip = [(y, x, v * (-1) ** ((y + x) % 2)) for y, x, v in parts]
    assert _error(tapered, lambda r: masked(r, (_waves(flip, r, 1) * _sign(r)).real)) <= BOUND
    grid = _fill(parts, -1)
    device.grid_to_image(G, grid, prol, work, image)
    ref = torch.zeros((G, G), dtype=torch.float64, device="cuda")
    for y, x, v in parts:
        cy, cx = (y + G // 2) % G, (x + G // 2) % G
        ref[cy, cx] += (-1) ** ((cy + cx) % 2) * v.real
    assert _error(lambda r: tapered(r) / G ** 2, lambda r: masked(r, ref[r])) <= BOUND
