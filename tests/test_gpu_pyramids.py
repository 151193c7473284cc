"""Intensity and depth pyramids where their tiles end.

The intensity pyramid makes three levels a launch in tiles of 32 x 32 pixels,
the depth pyramid every level of one launch in tiles of 64 x 16.  Against the
definition in FP32, one rounding per operation: equal, at the smallest level, at
sizes one off the tiles, with odd sizes on the way down and one to five levels,
widths with and without whole quads.  Vertices: level l's from its inverse depth within
four roundings (relative 2.4e-7 of their depth).
"""
from __future__ import annotations

import numpy as np
import pytest

from yetanotherslam_gb300 import rgbdfusion as rf

pytestmark = pytest.mark.gpu

CASES = [(4, 4, 1), (9, 8, 2), (32, 32, 2), (33, 31, 3), (65, 17, 3), (129, 95, 4), (255, 191, 5), (640, 481, 5)]
F = np.float32


def _down(a, h, w):
    k = [F(0.0625), F(0.25), F(0.375), F(0.25), F(0.0625)]

    def idx(n, m):
        i = np.abs(2 * np.arange(n)[:, None] + np.arange(-2, 3))
        return np.where(i >= m, 2 * (m - 1) - i, i)

    rows, cols = idx(h, a.shape[0]), idx(w, a.shape[1])
    s = np.zeros((h, a.shape[1]), F)
    for i in range(5):
        s = s + k[i] * a[rows[:, i]]
    out = np.zeros((h, w), F)
    for j in range(5):
        out = out + k[j] * s[:, cols[:, j]]
    return out


@pytest.mark.parametrize("w,h,levels", CASES)
def test_pyramids_match_the_definition(cuda, w, h, levels):
    rng = np.random.default_rng(w)
    gray = rng.integers(0, 256, (h, w), dtype=np.uint8)
    depth = rng.uniform(0.1, 9.0, (h, w)).astype(F)
    depth[rng.random((h, w)) < 0.3] = rng.choice([0.0, np.nan, np.inf, 0.2, 8.0])
    fx, cx, cy = 1.1 * w, 0.49 * w, 0.51 * h
    tr = rf.RGBDTracking(w, h, np.array([[fx, 0, cx], [0, fx, cy], [0, 0, 1.0]]), num_levels=levels)
    tr.SetTrackingImage(gray)
    tr.SetTrackingDepth(depth)
    tr.SetReferenceImage(gray)
    tr.SetReferenceDepth(depth)
    img = gray.astype(F)
    with np.errstate(all="ignore"):
        ok = (depth > F(0.2)) & (depth < F(8.0))
        inv = np.where(ok, F(1) / depth, F(0)).astype(F)
    for l in range(levels):
        wl, hl = w >> l, h >> l
        if l:
            img = _down(img, hl, wl)
            inv = inv[:2 * hl:2, :2 * wl:2].copy()
            inv[-1, :] = 0
            inv[:, -1] = 0
        gx, gy = np.zeros_like(img), np.zeros_like(img)
        gx[1:-1, 1:-1] = (img[1:-1, 2:] - img[1:-1, :-2]) * F(0.5)
        gy[1:-1, 1:-1] = (img[2:, 1:-1] - img[:-2, 1:-1]) * F(0.5)
        for which, want in ((0, img), (1, gx), (2, gy), (3, inv), (6, img), (7, inv)):
            assert np.array_equal(tr.level_buffer(l, which).numpy(), want), (l, which)
        z = 1.0 / np.where(inv > 0, inv, 1).astype(np.float64)
        near = np.abs(z - 3.0) < 1e-6  # the cut-off may fall on either side
        seen = (inv > 0) & (z < 3.0)
        y, x = np.mgrid[:hl, :wl]
        want = np.stack([z * (x - cx / 2**l) * 2**l / fx, z * (y - cy / 2**l) * 2**l / fx, z], -1)
        for which in (4, 8):
            v = tr.level_buffer(l, which).numpy()
            assert np.array_equal((v[..., 3] > 0) | near, seen | near), (l, which)
            both = seen & (v[..., 3] > 0)
            assert (np.abs(v[..., :3] - want)[both] <= 2.4e-7 * z[both][:, None] * 2).all(), (l, which)
        for v, n in ((4, 5), (8, 9)):
            a = tr.level_buffer(l, v).numpy()[..., 3] > 0
            good = np.zeros_like(a)
            good[:-1, :-1] = a[:-1, :-1] & a[:-1, 1:] & a[1:, :-1]
            assert np.array_equal(tr.level_buffer(l, n).numpy()[..., 3] > 0, good), (l, n)
