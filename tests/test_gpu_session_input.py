"""Where a session's frame comes from: device memory, host memory that the
frame's graph reads in place (aligned, pageable or pinned), or host memory that
is copied first (unaligned, or of an image whose bytes are no multiple of 16).
The same frames, so the same poses and raycasts bit for bit."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from tests.helpers import sequence
from yetanotherslam_gb300 import rgbdfusion as rf
from yetanotherslam_gb300 import synth

pytestmark = pytest.mark.gpu


def _host(a, how):
    if how == "device":
        return torch.from_numpy(a.view(np.uint8 if a.dtype == np.uint8 else np.int16)).cuda()
    if how == "pinned":
        t = torch.empty(a.shape, dtype=torch.uint8 if a.dtype == np.uint8 else torch.int16).pin_memory()
        v = t.numpy().view(a.dtype)
        v[...] = a
        return v
    room = np.zeros(a.nbytes + 64, np.uint8)
    at = -room.ctypes.data % 16 + (2 if how == "unaligned" else 0)
    v = room[at:at + a.nbytes].view(a.dtype).reshape(a.shape)
    v[...] = a
    return v


@pytest.mark.parametrize("w,h", [(160, 120), (97, 73), (320, 240)])
def test_every_source_gives_the_same_frames(cuda, w, h):
    seq = sequence(5, 5, w, h)
    want = None
    for how in ("device", "aligned", "unaligned", "pinned"):
        s = rf.Session(w, h, synth.intrinsics(w, h), hash_slots=1 << 18, max_blocks=1 << 16, voxel_size=0.008)
        got = []
        for rgb, depth, *_ in seq:
            r, d = _host(np.ascontiguousarray(rgb), how), _host(np.ascontiguousarray(depth), how)
            torch.cuda.synchronize()
            status, pose = s.process(r, d)
            got.append(pose.copy())
            assert status == 0
        s.close()
        if want is None:
            want = got
        for k, (a, b) in enumerate(zip(got, want)):
            assert np.array_equal(a, b), (how, k)


@pytest.mark.parametrize("w,h", [(64, 48), (61, 43), (1, 1), (637, 477)])
def test_host_depth_and_image_are_read_whole(cuda, w, h):
    """Fuse and the tracker's images from host memory, in place and copied: bytes
    that are no multiple of 16, and rows that do not adjoin."""
    rng = np.random.default_rng(w * h)
    z = rng.uniform(0.4, 2.5, (h, w)).astype(np.float32)
    gray = rng.integers(0, 256, (h, w)).astype(np.uint8)
    K = (0.9 * w, 0.9 * w, (w - 1) / 2, (h - 1) / 2)
    got = []
    for how in ("device", "aligned", "unaligned"):
        m = rf.MapStruct(K)
        m.create_config(1 << 18, 1 << 15, 0.02, 0.06, rf.VOXEL_F32)
        zz = torch.from_numpy(z).cuda() if how == "device" else _host(z, how) if how == "aligned" else None
        if zz is None:  # four bytes past a 16-byte boundary
            room = np.zeros(z.size + 8, np.float32)
            at = -room.ctypes.data % 16 // 4 + 1
            zz = room[at:at + z.size].reshape(z.shape)
            zz[...] = z
        torch.cuda.synchronize()
        m.Fuse(zz, np.eye(4))
        c, s, wt = m.export()
        order = np.lexsort(c.T)
        got.append((c[order], s[order], wt[order]))
        if min(w, h) >= 43:
            tr = rf.RGBDTracking(w, h, np.array([[K[0], 0, K[2]], [0, K[1], K[3]], [0, 0, 1]]), num_levels=2)
            tr.SetTrackingImage(torch.from_numpy(gray).cuda() if how == "device" else _host(gray, how))
            tr.SetTrackingDepth(zz)
            got[-1] += tuple(tr.level_buffer(l, q).numpy() for l in range(2) for q in range(6))
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a, b)
