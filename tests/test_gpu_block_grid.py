"""The raycast's block grid where it must not be believed: after its epochs wrap
and its cells are cleared, and when the map's blocks have changed between the
fusion that filled it and the raycast that reads it.  Every comparison is bit
for bit."""
from __future__ import annotations

import numpy as np
import pytest

from tests.helpers import rel_poses, sequence
from yetanotherslam_gb300 import rgbdfusion as rf
from yetanotherslam_gb300 import synth
from yetanotherslam_gb300.batching import Batch

pytestmark = pytest.mark.gpu

W, H, VS = 160, 120, 0.01


def _map(seed, frame):
    seq = sequence(seed, 4, W, H)
    m = rf.MapStruct(synth.intrinsics(W, H))
    m.create_config(1 << 16, 1 << 14, VS, 3 * VS, rf.VOXEL_F32)
    m.Fuse(seq[frame][2], rel_poses(seq)[frame])
    return m


def test_raycasts_across_the_epochs(cuda):
    """Two maps of different blocks in turn with one engine, past two wraps: a cell
    of the other map, or of 255 raycasts ago, would be a wrong block."""
    maps = [_map(7, 0), _map(8, 3)]
    want = []
    for m in maps:
        fresh = rf.RayTraceEngine(W, H, synth.intrinsics(W, H))
        fresh.RayTrace(m, np.eye(4))
        want.append(fresh.GetVMap().torch().clone())
        assert (want[-1][..., 3] > 0).any()
    engine = rf.RayTraceEngine(W, H, synth.intrinsics(W, H))
    got = engine.GetVMap().torch()
    for k in range(520):
        engine.RayTrace(maps[k % 2], np.eye(4))
        assert got.isnan().equal(want[k % 2].isnan()), k
        assert got.nan_to_num(5.0).equal(want[k % 2].nan_to_num(5.0)), k


def _permuted_again(m, seed):
    """The map's blocks in another pool order."""
    c, s, wt = m.export()
    order = np.random.default_rng(seed).permutation(len(c))
    assert len(c) > 100
    return c[order], s[order], wt[order]


def _reset_import(m, seed):
    blocks = _permuted_again(m, seed)
    m.Reset()
    m.import_blocks(*blocks)


def _swap(m, seed):
    other = rf.MapStruct(synth.intrinsics(W, H))
    other.create_config(1 << 16, 1 << 14, VS, 3 * VS, rf.VOXEL_F32)
    other.import_blocks(*_permuted_again(m, seed))
    m.Swap(other)


def _load(m, seed, path):
    other = rf.MapStruct(synth.intrinsics(W, H))
    other.create_config(1 << 16, 1 << 14, VS, 3 * VS, rf.VOXEL_F32)
    other.import_blocks(*_permuted_again(m, seed))
    other.SaveToFile(path)
    m.ReadFromFile(path)


def _import_more(m, seed):
    """Blocks that the grid covers and that no ray reaches before the surface: the
    block set is another one, the raycast the same."""
    c, s, wt = m.export()
    far = np.array([[0, 0, -2], [1, 0, -2]], np.int32)  # behind the camera
    m.import_blocks(far, s[:2], wt[:2])


EDITS = {"reset_import": _reset_import, "swap": _swap, "load": _load, "import_more": _import_more,
         "reserve": lambda m, seed: m.Reserve(1 << 17, 1 << 15)}


def _run(edit, how, tmp_path):
    seq = sequence(7, 6, W, H)
    s = rf.Session(W, H, synth.intrinsics(W, H), hash_slots=1 << 16, max_blocks=1 << 14, voxel_size=VS,
                   voxel_format=rf.VOXEL_F32, use_graph=how != "eager")
    batch = Batch([s]) if how == "batch" else None
    out = []
    for k, (rgb, depth, *_) in enumerate(seq):
        if edit and k in (2, 4):
            m = s.map()
            args = (str(tmp_path / "m.yas"),) if edit == "load" else ()
            EDITS[edit](m, k, *args)
        if batch:
            batch.step([(rgb, depth)])
            poses, status, _ = batch.wait()
            out.append((status[0], np.array(poses[0])))
        else:
            status, pose = s.process(rgb, depth)
            out.append((status, pose.copy()))
    m = s.map()
    c, sd, wt = m.export()
    order = np.lexsort(c.T)
    keep = slice(None)
    if edit == "import_more":
        keep = ~((c[order][:, 2] == -2) & (c[order][:, 1] == 0) & np.isin(c[order][:, 0], (0, 1)))
    out.append((c[order][keep], sd[order][keep], wt[order][keep]))
    if batch:
        batch.close()
    s.close()
    return out


@pytest.mark.parametrize("how", ["graph", "eager", "batch"])
@pytest.mark.parametrize("edit", sorted(EDITS))
def test_frames_after_the_maps_blocks_changed(cuda, edit, how, tmp_path):
    """A session whose map is rearranged between frames, without a voxel changed,
    tracks and fuses as one whose map is left alone."""
    want, got = _run(None, how, tmp_path), _run(edit, how, tmp_path)
    for k, (a, b) in enumerate(zip(want, got)):
        for x, y in zip(a, b):
            assert np.array_equal(x, y), k


@pytest.mark.parametrize("how", ["graph", "batch"])
def test_a_map_emptied_between_frames_is_a_miss(cuda, how):
    """No ray finds a block that was reset: nothing is left to track against with ICP."""
    seq = sequence(7, 4, W, H)
    s = rf.Session(W, H, synth.intrinsics(W, H), hash_slots=1 << 16, max_blocks=1 << 14, voxel_size=VS,
                   voxel_format=rf.VOXEL_F32)
    batch = Batch([s]) if how == "batch" else None

    def frame(rgb, depth):
        if batch:
            batch.step([(rgb, depth)])
            batch.wait()
        else:
            s.process(rgb, depth)

    tr = rf.RGBDTracking.__new__(rf.RGBDTracking)
    tr.handle = rf.C.c_void_p()
    rf.L.call("yas_session_tracker", s.handle, rf.C.byref(tr.handle))
    for rgb, depth, *_ in seq[:3]:
        frame(rgb, depth)
    s.map().Reset()
    frame(*seq[3][:2])
    sides = [tr.level_buffer(0, q).numpy()[..., 3] for q in (4, 8)]  # the frame's own vertices, and the model
    tr.handle = rf.C.c_void_p()
    assert sorted(bool((w > 0).any()) for w in sides) == [False, True]
    if batch:
        batch.close()
    s.close()
