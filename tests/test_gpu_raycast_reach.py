"""Raycast where its march takes another path: rays whose coordinates are too
large for the floors by a rounding sum, and cells that straddle the border of
the block grid, which look their neighbours up one by one.

A plane across the view, seen along z by a camera without rotation: the sdf is
linear in z and voxels are a power of two wide, so every quantity along z is
the same wherever the camera stands, and the vertex depth is the plane's.  The
interpolation, the two correction moves and the change of coordinates round a
few times each at up to 2^11 voxels, 2^-13 voxels a rounding: 10 roundings are
below 2^-9 voxels.
"""
from __future__ import annotations

import numpy as np
import pytest

from yetanotherslam_gb300 import rgbdfusion as rf

pytestmark = pytest.mark.gpu

W, H, F = 93, 71, 400.0


def _plane(vs, zv, shift_blocks, fmt):
    """Map of a plane at voxel z = zv, all blocks in view at it, moved by shift_blocks along x."""
    K = (F, F, (W - 1) / 2, (H - 1) / 2)
    half = int(np.ceil(zv * 0.5 * W / F / 8)) + 1
    n = 2 * half
    bx, by, bz = np.meshgrid(np.arange(-half, half), np.arange(-half, half), [zv // 8 - 1, zv // 8], indexing="ij")
    coords = np.stack([bx.ravel() + shift_blocks, by.ravel(), bz.ravel()], 1).astype(np.int32)
    z = coords[:, 2, None] * 8 + np.arange(512)[None] // 64
    sdf = np.clip((zv - z) / 3.0, -1, 1).astype(np.float32)
    m = rf.MapStruct(K)
    m.create_config(1 << 20, max(1 << 14, 2 * n * n + 64), vs, 3 * vs, fmt)
    m.import_blocks(coords, sdf, np.full(sdf.shape, 4, np.int32))
    return K, m


@pytest.mark.parametrize("fmt", [rf.VOXEL_F32, rf.VOXEL_F16])
@pytest.mark.parametrize("bits,zv,shift", [
    (6, 64, 0),  # near the origin
    (6, 64, 1 << 19),  # 2^22 voxels along x
    (6, 64, -(1 << 18)),  # 2^21: rays on both sides of the rule
    (9, 1152, 0),  # the plane on the far border of the block grid
    (9, 1152, 1 << 18),  # both
])
def test_plane_depth(cuda, fmt, bits, zv, shift):
    vs = 2.0 ** -bits
    K, m = _plane(vs, zv, shift, fmt)
    T = np.eye(4)
    T[0, 3] = shift * 8 * vs
    rc = rf.RayTraceEngine(W, H, K)
    rc.RayTrace(m, T)
    v = rc.GetVMap().numpy()
    assert (v[..., 3] > 0).all(), f"{int((v[..., 3] <= 0).sum())} pixels miss the plane"
    # F16 voxels keep thirds to 2^-19 of the truncation
    tol = vs * (2.0 ** -9 + (3 * 2.0 ** -17 if fmt == rf.VOXEL_F16 else 0))
    assert np.abs(v[..., 2] - zv * vs).max() <= tol
