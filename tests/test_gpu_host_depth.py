"""Fuse and Defuse of a host depth: rows that do not adjoin, and what has been done
when the call returns."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from yetanotherslam_gb300 import _lib as L
from yetanotherslam_gb300 import rgbdfusion as rf

pytestmark = pytest.mark.gpu


def _map(K, stream=None, vs=0.02):
    m = rf.MapStruct(K, stream)
    m.create_config(1 << 18, 1 << 15, vs, 3 * vs, rf.VOXEL_F32)
    return m


def _blocks(m):
    c, s, wt = m.export()
    order = np.lexsort(c.T)
    return c[order], s[order], wt[order]


@pytest.mark.parametrize("w,h,pad", [(64, 48, 5), (61, 43, 3), (61, 43, 64), (7, 1, 9)])
def test_padded_rows_fuse_as_adjoining_ones(cuda, w, h, pad):
    z = np.random.default_rng(w + pad).uniform(0.4, 2.5, (h, w)).astype(np.float32)
    # the last row ends the allocation: what would be its padding is not there
    room = np.zeros(h * (w + pad) - pad + 4, np.float32)
    at = -room.ctypes.data % 16 // 4  # an aligned image, as the in-place read takes
    rows = np.lib.stride_tricks.as_strided(room[at:], (h, w), (4 * (w + pad), 4))
    rows[...] = z
    K = (0.9 * w, 0.9 * w, (w - 1) / 2, (h - 1) / 2)
    one, two = _map(K), _map(K)
    T = L.pose_from(np.eye(4))
    for name in ("yas_map_fuse_depth", "yas_map_fuse_depth", "yas_map_defuse_depth"):
        L.call(name, one.handle, z.ctypes.data, w, h, 4 * w, 0, C.byref(T))
        L.call(name, two.handle, room[at:].ctypes.data, w, h, 4 * (w + pad), 0, C.byref(T))
        for a, b in zip(_blocks(one), _blocks(two)):
            assert np.array_equal(a, b)


def test_a_host_depth_is_fused_when_the_call_returns(cuda):
    """The map's stream has nothing left to do: a program that reads the map on
    another stream, or looks for an error, need not wait first."""
    stream = torch.cuda.Stream()
    w, h = 1280, 720
    z = np.random.default_rng(3).uniform(0.8, 2.5, (h, w)).astype(np.float32)
    m = _map((0.9 * w, 0.9 * w, (w - 1) / 2, (h - 1) / 2), stream.cuda_stream)
    for _ in range(3):
        m.Fuse(z, np.eye(4))
        assert stream.query()
        m.Defuse(z, np.eye(4))
        assert stream.query()


def test_a_call_that_fails_after_its_read_was_enqueued_waits_for_it(cuda):
    """More rows than a launch's grid takes: the host refuses the allocation pass
    when the depth's read is already under way."""
    stream = torch.cuda.Stream()
    w, h = 64, 8 * 65535 + 8
    z = np.full((h, w), np.float32(0.5))
    m = _map((0.9 * w, 0.9 * w, (w - 1) / 2, (h - 1) / 2), stream.cuda_stream)
    m.Fuse(z[:8], np.eye(4))
    with pytest.raises(L.YasError):
        m.Fuse(z, np.eye(4))
    assert stream.query()
