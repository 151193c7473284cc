"""Marching cubes from rows of bits, and the canvas's queue of triangles.

Meshes: random blocks (every case, unobserved voxels, missing neighbours,
negative coordinates) in every voxel format against the table applied cube by
cube: cubes and cases equal; a soup cut off by its capacity is the whole one's
beginning, bit for bit.  Canvas: bit-exact against the oracle at triangle counts
around a warp's queue and at sizes from below a pixel to most of the image.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import oracle
from yetanotherslam_gb300 import _lib as L
from yetanotherslam_gb300 import rgbdfusion as rf

pytestmark = pytest.mark.gpu

K = (100.0, 100.0, 48.0, 36.0)
CORNERS = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]


def _expected(m):
    """Sorted rows (x, y, z, case), one per triangle."""
    count = np.zeros(256, np.uint8)
    L.load().yas_mc_tables(None, None, count.ctypes.data_as(C.c_void_p))
    coords, sdf, wt = m.export()
    lo = coords.min(0)
    n = (coords.max(0) - lo + 2) * 8
    val = np.full(n, np.nan, np.float32)  # by x, y, z
    for c, s, w in zip(coords - lo, sdf, wt):
        a, b, d = c * 8
        val[a:a + 8, b:b + 8, d:d + 8] = np.where(w > 0, s, np.nan).reshape(8, 8, 8).transpose(2, 1, 0)
    at = [val[x:n[0] - 1 + x, y:n[1] - 1 + y, z:n[2] - 1 + z] for x, y, z in CORNERS]
    seen = np.all([~np.isnan(a) for a in at], 0)
    case = sum((a < 0).astype(int) << i for i, a in enumerate(at))
    tris = np.where(seen, count[case], 0)
    xyz = np.argwhere(tris > 0)
    rows = np.column_stack([xyz + lo * 8, case[tuple(xyz.T)]])
    return rows[np.lexsort(rows.T)].repeat(tris[tuple(xyz.T)][np.lexsort(rows.T)], 0)


@pytest.mark.parametrize("fmt", [rf.VOXEL_F32, rf.VOXEL_F16, rf.VOXEL_S24, rf.VOXEL_S16])
@pytest.mark.parametrize("blocks", [1, 2, 60])
def test_random_blocks(cuda, fmt, blocks):
    rng = np.random.default_rng(blocks)
    coords = np.unique(rng.integers(-2, 3, (blocks, 3)), axis=0).astype(np.int32)
    sdf = rng.uniform(-1, 1, (len(coords), 512)).astype(np.float32)
    wt = (rng.random((len(coords), 512)) < 0.95).astype(np.float32) * 3
    m = rf.MapStruct(K)
    m.create_config(1 << 12, 1 << 10, 0.01, 0.03, fmt)
    m.import_blocks(coords, sdf, wt)
    pts, nrm, cases, cube = rf.MeshEngine(400_000).Meshify(m)
    rows = np.column_stack([cube, cases])
    want = _expected(m)
    assert len(want) > 100 and np.array_equal(rows[np.lexsort(rows.T)], want)
    cut = len(pts) // 2 + 1
    me = rf.MeshEngine(cut)
    p, n, c, x = me.Meshify(m)
    assert me.overflow and len(p) == cut
    assert np.array_equal(p, pts[:cut]) and np.array_equal(n, nrm[:cut])
    assert np.array_equal(c, cases[:cut]) and np.array_equal(x, cube[:cut])


@pytest.mark.parametrize("n", [1, 31, 32, 33, 129, 4097])
@pytest.mark.parametrize("size", [0.002, 0.03, 0.8])
def test_canvas_queue(cuda, n, size):
    w, h = 97, 73
    rng = np.random.default_rng(n)
    centre = rng.uniform([-0.6, -0.5, -0.1], [0.6, 0.5, 1.5], (n, 1, 3))
    pts = (centre + rng.uniform(-size, size, (n, 3, 3))).astype(np.float32).reshape(n, 9)
    nrm = rng.normal(size=(n, 3, 3))
    nrm = (nrm / np.linalg.norm(nrm, axis=-1, keepdims=True)).astype(np.float32).reshape(n, 9)
    cv = rf.Canvas(w, h, K)
    cv.draw_triangles(pts, nrm, np.eye(4), np.eye(4))
    rgba, depth = cv.read()
    want = oracle.canvas_resolve(oracle.canvas_draw(pts, nrm, np.eye(4), np.eye(4), K, w, h))
    assert np.array_equal(rgba, want[0]) and np.array_equal(depth, want[1])
