"""What the raycast's block grid costs in memory: nothing until a raycaster's first
raycast, and no session refused for it.  Without one a raycast takes its blocks from
the hash table, the same bits."""
from __future__ import annotations

import gc
import threading
import time

import numpy as np
import pytest
import torch

from tests.helpers import sequence
from yetanotherslam_gb300 import _lib as L
from yetanotherslam_gb300 import rgbdfusion as rf
from yetanotherslam_gb300 import serving, synth

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _free():
    gc.collect()
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_raycasters_that_do_not_raycast_hold_no_grid(cuda):
    K = synth.intrinsics(160, 120)
    keep = [rf.RayTraceEngine(160, 120, K)]
    before = _free()
    keep += [rf.RayTraceEngine(160, 120, K) for _ in range(16)]
    assert before - _free() < 16 * 2 * MB  # images and tiles: 0.5 MB each


def _estimate(w, h, levels, slots, blocks):
    """The server's own footprint of a session with 4-byte voxels, without a grid."""
    px = sum((w >> l) * (h >> l) for l in range(levels))
    return slots * 16 + blocks * (12 + 512 * 4) + 88 * px + 49 * w * h + 8 * MB


def _serve(srv, sids, seq):
    out = []
    for rgb, depth, *_ in seq:
        for sid in sids:
            assert srv.submit(sid, rgb, depth) == 0
        srv.drain()
        got = sorted(srv.poll(), key=lambda r: r["session"])
        assert [r["status"] for r in got] == [0] * len(sids)
        out.append([r["Tcm"] for r in got])
    return out


@pytest.mark.parametrize("sessions", [1, 2])
def test_no_session_is_refused_for_its_grid(cuda, sessions):
    """Room for the sessions and 6 MB, less than a grid: the first of two takes one and gives
    it back for the second."""
    w, h, kw = 160, 120, dict(hash_slots=1 << 20, max_blocks=1 << 17, voxel_size=0.004, num_levels=3)
    seq, K = sequence(7, 4, w, h), synth.intrinsics(w, h)
    roomy = serving.Server(hbm_reserve_bytes=1 << 30)
    ids = [roomy.open(w, h, K, **kw) for _ in range(sessions)]
    want = _serve(roomy, ids, seq)
    roomy.close()

    need = _estimate(w, h, 3, 1 << 20, 1 << 17)
    probe = serving.Server(hbm_reserve_bytes=1 << 30)
    before = _free()
    sid = probe.open(w, h, K, **kw)
    own = before - _free()  # what a session with its grid takes in fact
    probe.close_session(sid)
    probe.close()
    held = (sessions - 1) * (own - 17 * MB)
    tight = serving.Server(hbm_reserve_bytes=_free() - held - need - 6 * MB)
    ids = [tight.open(w, h, K, **kw)]
    got = _serve(tight, ids, seq[:2])
    for _ in range(1, sessions):
        ids.append(tight.open(w, h, K, **kw))
    if sessions == 1:
        got += _serve(tight, ids, seq[2:])
        assert all(np.array_equal(a, b) for x, y in zip(got, want) for a, b in zip(x, y))
    else:  # the first goes on without its grid, the second starts
        for k, (rgb, depth, *_) in enumerate(seq[2:]):
            tight.submit(ids[0], rgb, depth)
            tight.submit(ids[1], *seq[k][:2])
            tight.drain()
            r = sorted(tight.poll(), key=lambda r: r["session"])
            assert np.array_equal(r[0]["Tcm"], want[k + 2][0]) and np.array_equal(r[1]["Tcm"], want[k][1])
    tight.close()


def test_a_busy_session_gives_its_grid_back(cuda):
    """Its queue does not empty while another session is opened: that one waits for a
    frame, not for the queue."""
    w, h, kw = 160, 120, dict(hash_slots=1 << 20, max_blocks=1 << 17, voxel_size=0.004, num_levels=3)
    seq, K = sequence(7, 4, w, h), synth.intrinsics(w, h)
    need = _estimate(w, h, 3, 1 << 20, 1 << 17)
    probe = serving.Server(hbm_reserve_bytes=1 << 30)
    before = _free()
    own = (probe.open(w, h, K, **kw), before - _free())[1]
    probe.close()
    srv = serving.Server(hbm_reserve_bytes=_free() - (own - 17 * MB) - need - 6 * MB)
    first = srv.open(w, h, K, **kw)
    walk = [0, 1, 2, 3, 2, 1]
    stop, sent = threading.Event(), [0]

    def feed():
        while not stop.is_set():
            if srv.submit(first, *seq[walk[sent[0] % 6]][:2]) == 0:
                sent[0] += 1

    t = threading.Thread(target=feed)
    t.start()
    try:
        while sent[0] < 200:
            time.sleep(0.001)
        since = time.monotonic()
        second = srv.open(w, h, K, **kw)
        took = time.monotonic() - since
    finally:
        stop.set()
        t.join()
    assert took < 5.0
    assert srv.submit(second, *seq[0][:2]) == 0
    srv.drain()
    assert sum(r["session"] == first and r["status"] == 0 for r in srv.poll(1 << 16)) == sent[0]
    srv.close()


def test_a_session_that_cannot_fit_costs_nobody_a_grid(cuda):
    srv = serving.Server(hbm_reserve_bytes=1 << 30)
    srv.open(160, 120, synth.intrinsics(160, 120), hash_slots=1 << 16, max_blocks=1 << 12, voxel_size=0.01)
    before = _free()
    with pytest.raises(L.YasError):
        srv.open(160, 120, synth.intrinsics(160, 120), hash_slots=1 << 20, max_blocks=1 << 29, voxel_size=0.01)
    assert _free() == before
    srv.close()
