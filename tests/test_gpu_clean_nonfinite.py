"""Hogbom with deferred tile updates on NaN and infinite samples and on equal
peaks, against the oracle, bit for bit (NaN equal to NaN).  The PSF's bad
samples lie next to large finite ones, whose effect decides the next
component: a tile's bound has to count them although the block maximum is a
NaN, whatever the NaN's bits.  With the final residual (G > 2752, device entry
point) and without (G >= 1536, actor)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NANS = {"nan_ffff": 0x7fffffff, "nan_quiet": 0x7fc00000, "nan_signed": 0xffffffff, "nan_small": 0x7f800001,
        "inf": 0x7f800000, "-inf": 0xff800000}


def _point_psf(G):
    yy, xx = np.mgrid[-4:5, -4:5]
    psf = np.zeros((G, G), np.float32)
    psf[G // 2 - 4:G // 2 + 5, G // 2 - 4:G // 2 + 5] = np.exp(-(yy ** 2 + xx ** 2) / 4.0)
    return psf


def _sky(G, seed, n=30):
    rng = np.random.default_rng(seed)
    res = (0.001 * rng.standard_normal((G, G))).astype(np.float32)
    for y, x in rng.integers(G // 5, 4 * G // 5, (n, 2)):
        res[y, x] += np.float32(rng.uniform(0.3, 0.6))
    return res


def _same(a, b):
    """Equal bits, any NaN equal to any other."""
    a, b = np.asarray(a, np.float32), np.asarray(b, np.float32)
    assert a.shape == b.shape
    same = (a.view(np.uint32) == b.view(np.uint32)) | (np.isnan(a) & np.isnan(b))
    assert same.all(), (int((~same).sum()), np.argwhere(~same)[:3])


def _compare(sdp, device, actors, oracle, res, psf, minor, psf_max=1.0):
    import torch
    G = res.shape[0]
    res, psf = np.ascontiguousarray(res).reshape(-1), np.ascontiguousarray(psf).reshape(-1)
    n1, s1, m1, r1 = oracle.hogbom(G, minor, minor, res, psf, psf_max, 1e-5, weak=0.0)
    if G <= 2752:
        cfg = sdp.make_config(G, 1.0, 1.0, psf_max_value=psf_max, cell_size=1e-5, weak_source_percent_img=0.0)
        n2, s2, m2 = actors.hogbom(cfg, G, minor, minor, res, psf)
        r2 = r1
    else:
        params = sdp.CleanParams(G, minor, minor, 0.1, 1.5, 0.0, psf_max, 1e-5)
        r, p = torch.from_numpy(res.copy()).cuda(), torch.from_numpy(psf).cuda()
        m = torch.zeros(G * G, dtype=torch.float32, device="cuda")
        s = torch.zeros((minor, 3), dtype=torch.float32, device="cuda")
        c = torch.zeros(1, dtype=torch.int32, device="cuda")
        ws = torch.empty(device.hogbom_workspace_bytes(G), dtype=torch.uint8, device="cuda")
        device.hogbom(params, r, p, m, s, c, ws)
        n2 = int(c.item())
        s2, m2, r2 = s[:n2].cpu().numpy(), m.cpu().numpy(), r.cpu().numpy()
    assert n1 == n2 == minor
    _same(s2, s1)
    _same(m2, m1)
    _same(r2, r1)
    return s1


@pytest.mark.parametrize("kind", sorted(NANS))
@pytest.mark.parametrize("G", [1536, 2784])
def test_bad_psf_samples(sdp, device, actors, oracle32, G, kind):
    """A bad sample beside sidelobes of -12: the subtraction of a component
    raises the sidelobe's pixels above every other (mirrored in x)."""
    psf = _point_psf(G)
    h = G // 2
    for dy, dx in ((70, 90), (-200, 33)):
        psf[h + dy, h + dx] = -12.0
        psf.view(np.uint32)[h + dy + 3, h + dx + 5] = NANS[kind]
    _compare(sdp, device, actors, oracle32, _sky(G, 3), psf, 12)


@pytest.mark.parametrize("kind", sorted(NANS))
@pytest.mark.parametrize("G", [1536, 2784])
def test_bad_pixels(sdp, device, actors, oracle32, G, kind):
    """Bad samples in the dirty image: the first pixel, one on a tile's edge, one inside."""
    res, psf = _sky(G, 4), _point_psf(G)
    for y, x in ((0, 0), (640, 671), (900, 1001)):
        res.view(np.uint32)[y, x] = NANS[kind]
    _compare(sdp, device, actors, oracle32, res, psf, 8)


@pytest.mark.parametrize("G", [1536, 2784])
def test_equal_peaks(sdp, device, actors, oracle32, G):
    """Peaks of equal size, of both signs, in one tile and in others: the
    smaller index goes first.  The gain brings each down by the same factor,
    so ties come back in every round."""
    res, psf = np.zeros((G, G), np.float32), _point_psf(G)
    spots = [(G - 9, 40), (100, 1200), (100, 1215), (115, 1200), (700, 5), (701, 300), (12, 12)]
    for k, (y, x) in enumerate(spots):
        res[y, x] = -1.0 if k % 3 == 1 else 1.0
    s = _compare(sdp, device, actors, oracle32, res, psf, 30)
    first = [(int(round(float(y) / 1e-5)) + G // 2, int(round(float(x) / 1e-5)) + G // 2) for x, y, _ in s[:len(spots)]]
    assert first == sorted(spots)


def test_infinite_psf_max(sdp, device, actors, oracle32):
    """An infinite PSF maximum: the scale is zero, zero times infinity a NaN
    inside the component's window, and nothing changes outside it."""
    res = _sky(2784, 6)
    res[3, 5] = 2.0
    _compare(sdp, device, actors, oracle32, res, _point_psf(2784), 1, psf_max=float("inf"))


def test_negative_zeros(sdp, device, actors, oracle32):
    """Zeros keep their sign outside a component's window, also under a
    negative component (-0 - (-0) is +0)."""
    res, psf = _sky(2784, 7), _point_psf(2784)
    res[np.abs(res) < 0.01] = -0.0
    res[5, 7] = -2.0
    _compare(sdp, device, actors, oracle32, res, psf, 6)
