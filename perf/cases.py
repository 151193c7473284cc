"""The calls that programs make of this framework, as cases to be timed.

A case is one of these uses, over the sizes, voxel sizes, storage formats and
options that programs pass:

  session      one frame of a SLAM session (``Session.process``): tracking
               against the raycast map, then fusion
  batch        one step of several keyframe submaps (``Batch.step``/``wait``)
  served       one frame of each of several sessions through the request server
  fuse_raycast a depth frame at a known pose fused into a map
               (``MapStruct.Fuse``), and the map raycast from the next pose
  reintegrate  depth frames taken out of a map at their old poses and fused
               again at corrected ones (``Defuse``, ``Fuse``), and the result
               raycast: what follows a loop closure
  track        frame-to-frame tracking with ``RGBDTracking`` alone
  pyramids     a tracker's per-frame image and depth pyramids
  mesh_view    a saved submap's surface extracted into the caller's
               arrays (``yas_mesher_*``) and drawn into a viewer's image (``Canvas``)

Frames are rendered from seeded synthetic scenes (``synth.Scene``), as in the
tests and the benchmark; a session walks its frames back and forth, so its
motion stays smooth however often it is called.
"""
from __future__ import annotations

import os
import tempfile

import numpy as np
import torch

from yetanotherslam_gb300 import rgbdfusion as rf
from yetanotherslam_gb300 import synth
from yetanotherslam_gb300.batching import Batch
from yetanotherslam_gb300.serving import Server

FORMATS = {"f32": rf.VOXEL_F32, "f16": rf.VOXEL_F16, "s24": rf.VOXEL_S24, "s16": rf.VOXEL_S16}
MODES = {"rgb": rf.TRACK_RGB, "icp": rf.TRACK_ICP, "rgbd": rf.TRACK_RGBD}
ITERATIONS = (10, 5, 3, 3, 3)
MAX_TRIANGLES = 1_500_000


def listed():
    return [
        # a robot's small session: host frames as a camera driver hands them over
        {"name": "session_320x240_8mm_f32_host", "use": "session", "w": 320, "h": 240, "vs": 0.008, "fmt": "f32",
         "mode": "rgbd", "host": True},
        # the benchmark's session
        {"name": "session_640x480_5mm_f16", "use": "session", "w": 640, "h": 480, "vs": 0.005, "fmt": "f16",
         "mode": "rgbd", "host": False},
        # the large-map session
        {"name": "session_1280x720_4mm_f16", "use": "session", "w": 1280, "h": 720, "vs": 0.004, "fmt": "f16",
         "mode": "rgbd", "host": False},
        # keyframe submaps of uneven size, stepped together
        {"name": "batch_8_mixed_f16", "use": "batch", "n": 8, "vs": 0.005, "fmt": "f16"},
        # concurrent clients of the request server
        {"name": "served_8_mixed_f16", "use": "served", "n": 8, "vs": 0.005, "fmt": "f16"},
        # the smallest mapping calls: latency and launches
        {"name": "fuse_raycast_160x120_1cm_f32", "use": "fuse_raycast", "w": 160, "h": 120, "vs": 0.01, "fmt": "f32",
         "host": False},
        # mapping with known poses, an odd image size, the reference's voxel word, host depth
        {"name": "fuse_raycast_637x477_8mm_s16_host", "use": "fuse_raycast", "w": 637, "h": 477, "vs": 0.008,
         "fmt": "s16", "host": True},
        # re-integration after a pose correction
        {"name": "reintegrate_640x480_5mm_f16", "use": "reintegrate", "w": 640, "h": 480, "vs": 0.005, "fmt": "f16",
         "frames": 6},
        # visual odometry with the reference's five levels
        {"name": "track_640x480_rgbd_5_levels_host", "use": "track", "w": 640, "h": 480, "levels": 5, "mode": "rgbd",
         "host": True},
        # depth-only tracking of a small, odd image
        {"name": "track_333x251_icp_3_levels", "use": "track", "w": 333, "h": 251, "levels": 3, "mode": "icp",
         "host": False},
        # preprocessing of a frame
        {"name": "pyramids_640x480_3_levels", "use": "pyramids", "w": 640, "h": 480, "levels": 3},
        # a viewer shows a finished submap
        {"name": "mesh_view_640x480_6mm_f16", "use": "mesh_view", "w": 640, "h": 480, "vs": 0.006, "fmt": "f16",
         "frames": 6},
    ]


def _size(rng, lo, hi):
    """Image width (log-uniform, any parity) and height at a camera's aspect ratio."""
    w = int(round(lo * (hi / lo) ** rng.random()))
    return w, int(round(w * rng.choice((0.75, 0.75, 0.5625, 0.667)))) + rng.choice((0, 0, 1))


def draw(rng):
    use = rng.choice(("session", "session", "fuse_raycast", "fuse_raycast", "reintegrate", "track", "track", "batch",
                      "pyramids", "mesh_view"))
    w, h = _size(rng, 160, {"reintegrate": 800, "mesh_view": 640}.get(use, 1280))
    vs = round(0.004 * (0.01 / 0.004) ** rng.random(), 4)
    fmt = rng.choice(("f16", "f16", "f32", "s24", "s16"))
    if use == "session":
        return {"use": use, "w": w, "h": h, "vs": vs, "fmt": fmt, "mode": rng.choice(("rgbd", "rgbd", "icp")),
                "host": rng.random() < 0.5}
    if use == "batch":
        return {"use": use, "n": rng.randint(2, 8), "vs": max(vs, 0.005), "fmt": fmt}
    if use == "fuse_raycast":
        return {"use": use, "w": w, "h": h, "vs": vs, "fmt": fmt, "host": rng.random() < 0.5}
    if use == "reintegrate":
        return {"use": use, "w": w, "h": h, "vs": max(vs, 0.005), "fmt": fmt, "frames": rng.randint(2, 6)}
    if use == "track":
        return {"use": use, "w": w, "h": h, "levels": rng.randint(2, 5), "mode": rng.choice(("rgbd", "rgbd", "rgb", "icp")),
                "host": rng.random() < 0.5}
    if use == "pyramids":
        return {"use": use, "w": w, "h": h, "levels": rng.randint(2, 5)}
    return {"use": use, "w": w, "h": h, "vs": max(vs, 0.006), "fmt": fmt, "frames": rng.randint(2, 6)}


# ---------------------------------------------------------------- inputs
def _scene(seed):
    for k in range(16):  # a few seeds leave no room for their objects
        try:
            return synth.Scene(seed=1 + (int(seed) * 7919 + k) % 1000003)
        except RuntimeError:
            continue
    raise RuntimeError("no scene for this seed")


def _frames(seed, n, w, h):
    """n frames of a scene and their camera poses in the first frame's coordinates."""
    frames = _scene(seed).frames(n, w, h)
    first = np.linalg.inv(frames[0].Twc)
    return frames, [first @ f.Twc for f in frames]


def _metres(frame):
    return frame.depth.astype(np.float32) * np.float32(0.001)


def _walk(k, n):
    """Frame k of a walk back and forth over n frames."""
    k %= 2 * (n - 1)
    return k if k < n else 2 * (n - 1) - k


def _rgbd(frame, host):
    if host:
        return frame.rgb, frame.depth
    return torch.from_numpy(frame.rgb).cuda(), torch.from_numpy(frame.depth.view(np.int16)).cuda()


def _capacity(vs):
    """Hash slots and pool blocks of a map, as the configurations size them."""
    return (1 << 20, 1 << 17) if vs >= 0.0055 else (1 << 21, 1 << 18)


def _map(K, vs, fmt):
    slots, blocks = _capacity(vs)
    m = rf.MapStruct(K)
    m.create_config(slots, blocks, vs, 3 * vs, FORMATS[fmt])
    return m


def _session(w, h, vs, fmt, mode="rgbd"):
    slots, blocks = _capacity(vs)
    return rf.Session(w, h, synth.intrinsics(w, h), hash_slots=slots, max_blocks=blocks, voxel_size=vs,
                      voxel_format=FORMATS[fmt], mode=MODES[mode], num_levels=3, iterations=ITERATIONS)


def _sizes(n):
    """The resolutions of n sessions that run together."""
    return [((320, 240), (640, 480), (480, 360))[i % 3] for i in range(n)]


# ---------------------------------------------------------------- session
def _prepare_session(c, seed):
    n = 8
    frames, _ = _frames(seed, n, c["w"], c["h"])
    s = {"session": _session(c["w"], c["h"], c["vs"], c["fmt"], c["mode"]),
         "frames": [_rgbd(f, c["host"]) for f in frames], "k": 0}
    torch.cuda.synchronize()
    for _ in range(4):  # a session that is under way
        _run_session(s)
    # the vertex and normal maps that a frame's raycast leaves for the tracker, in turn
    tr = rf.RGBDTracking.__new__(rf.RGBDTracking)
    tr.handle, tr.session = rf.C.c_void_p(), s["session"]  # the maps keep their session alive
    rf.L.call("yas_session_tracker", s["session"].handle, rf.C.byref(tr.handle))
    s["model"] = [None, None]
    for _ in range(2):
        _run_session(s)
        s["model"][s["k"] & 1] = [tr.level_buffer(0, q).torch() for q in (4, 5)]
    tr.handle = rf.C.c_void_p()  # the session owns its tracker
    return s


def _run_session(s):
    status, pose = s["session"].process(*s["frames"][_walk(s["k"], len(s["frames"]))])
    s["k"] += 1
    return {"status": status, "pose": pose, "model": s["model"][s["k"] & 1] if "model" in s else None}


# ---------------------------------------------------------------- batch
def _prepare_batch(c, seed):
    sizes = _sizes(c["n"])
    sessions = [_session(w, h, c["vs"] if i % 2 else max(c["vs"], 0.008), c["fmt"]) for i, (w, h) in enumerate(sizes)]
    frames = [[_rgbd(f, False) for f in _frames(seed + 100 * i, 4, w, h)[0]] for i, (w, h) in enumerate(sizes)]
    torch.cuda.synchronize()
    s = {"batch": Batch(sessions), "frames": frames, "k": 0}
    for _ in range(4):
        _run_batch(s)
    return s


def _run_batch(s):
    s["batch"].step([f[_walk(s["k"], len(f))] for f in s["frames"]])
    poses, status, _ = s["batch"].wait()
    s["k"] += 1
    return {"poses": poses, "status": status}


# ---------------------------------------------------------------- served
def _prepare_served(c, seed):
    sizes = _sizes(c["n"])
    server = Server(max_sessions=c["n"])
    slots, blocks = _capacity(c["vs"])
    ids = [server.open(w, h, synth.intrinsics(w, h), hash_slots=slots, max_blocks=blocks, voxel_size=c["vs"],
                       voxel_format=FORMATS[c["fmt"]], num_levels=3, iterations=ITERATIONS) for w, h in sizes]
    frames = [_frames(seed + 100 * i, 4, w, h)[0] for i, (w, h) in enumerate(sizes)]
    s = {"server": server, "ids": ids, "frames": frames, "k": 0}
    for _ in range(4):
        _run_served(s)
    return s


def _run_served(s):
    for sid, f in zip(s["ids"], s["frames"]):
        fr = f[_walk(s["k"], len(f))]
        s["server"].submit(sid, fr.rgb, fr.depth)
    s["server"].drain()
    s["k"] += 1
    got = sorted(s["server"].poll(), key=lambda r: r["session"])
    return {"poses": np.stack([r["Tcm"] for r in got]), "status": np.array([r["status"] for r in got])}


# ---------------------------------------------------------------- mapping
def _prepare_fuse_raycast(c, seed):
    frames, poses = _frames(seed, 5, c["w"], c["h"])
    K = synth.intrinsics(c["w"], c["h"])
    depth = [_metres(f) for f in frames]
    if not c["host"]:
        depth = [torch.from_numpy(d).cuda() for d in depth]
        torch.cuda.synchronize()
    s = {"map": _map(K, c["vs"], c["fmt"]), "engine": rf.RayTraceEngine(c["w"], c["h"], K), "depth": depth,
         "poses": poses, "k": 0}
    s["vmap"] = s["engine"].GetVMap().torch()
    for _ in range(4):
        _run_fuse_raycast(s)
    return s


def _run_fuse_raycast(s):
    i, j = _walk(s["k"], len(s["poses"])), _walk(s["k"] + 1, len(s["poses"]))
    s["map"].Fuse(s["depth"][i], s["poses"][i])
    s["engine"].RayTrace(s["map"], s["poses"][j])
    s["k"] += 1
    return {"vertices": s["vmap"], "visible": s["engine"].GetNumVisibleBlock()}


def _turned(T, seed):
    """T moved by a loop closure's correction: a centimetre and half a degree."""
    r = np.random.default_rng(seed)
    w = r.normal(size=3)
    w *= np.radians(0.5) / np.linalg.norm(w)
    W = np.array([[0, -w[2], w[1]], [w[2], 0, -w[0]], [-w[1], w[0], 0]])
    C = np.eye(4)
    u, _, v = np.linalg.svd(np.eye(3) + W)
    C[:3, :3] = u @ v
    C[:3, 3] = r.normal(size=3) * 0.006
    return C @ T


def _prepare_reintegrate(c, seed):
    frames, poses = _frames(seed, c["frames"], c["w"], c["h"])
    K = synth.intrinsics(c["w"], c["h"])
    s = {"map": _map(K, c["vs"], c["fmt"]), "engine": rf.RayTraceEngine(c["w"], c["h"], K),
         "depth": [torch.from_numpy(_metres(f)).cuda() for f in frames], "old": poses,
         "new": [_turned(T, seed) for T in poses]}
    s["vmap"] = s["engine"].GetVMap().torch()
    for d, T in zip(s["depth"], s["old"]):
        s["map"].Fuse(d, T)
    return s


def _run_reintegrate(s):
    for d, a, b in zip(s["depth"], s["old"], s["new"]):
        s["map"].Defuse(d, a)
        s["map"].Fuse(d, b)
    s["engine"].RayTrace(s["map"], s["new"][-1])
    s["old"], s["new"] = s["new"], s["old"]  # the next correction takes them back
    return {"vertices": s["vmap"], "visible": s["engine"].GetNumVisibleBlock()}


# ---------------------------------------------------------------- tracking
def _gray(frame):
    return synth.gray_of(frame.rgb)


def _prepare_track(c, seed):
    n = 6
    frames, _ = _frames(seed, n, c["w"], c["h"])
    images = [(_gray(f), _metres(f)) for f in frames]
    if not c["host"]:
        images = [(torch.from_numpy(g).cuda(), torch.from_numpy(d).cuda()) for g, d in images]
    fx, fy, cx, cy = synth.intrinsics(c["w"], c["h"])
    K = np.array([[fx, 0, cx], [0, fy, cy], [0, 0, 1]])
    tr = rf.RGBDTracking(c["w"], c["h"], K, bRGB="rgb" in c["mode"], bIcp=c["mode"] != "rgb",
                         num_levels=c["levels"], iterations=ITERATIONS)
    s = {"tracker": tr, "images": images, "k": 0}
    tr.SetTrackingImage(images[0][0])
    tr.SetTrackingDepth(images[0][1])
    tr.SwapFrameBuffer()
    s["k"] = 1
    for _ in range(3):
        _run_track(s)
    return s


def _run_track(s):
    gray, depth = s["images"][_walk(s["k"], len(s["images"]))]
    s["tracker"].SetTrackingImage(gray)
    s["tracker"].SetTrackingDepth(depth)
    s["k"] += 1
    return {"transform": s["tracker"].GetTransform(None, True)}


def _fine_depth(frame, seed):
    """The frame's depth in metres with the sensor's sub-millimetre part."""
    z = frame.depth.astype(np.float32) * np.float32(0.001)
    part = np.random.default_rng(seed).uniform(-4e-4, 4e-4, z.shape).astype(np.float32)
    return np.where(z > 0, z + part, np.float32(0)).astype(np.float32)


def _prepare_pyramids(c, seed):
    frame = _scene(seed).render(0, c["w"], c["h"])
    fx, fy, cx, cy = synth.intrinsics(c["w"], c["h"])
    tr = rf.RGBDTracking(c["w"], c["h"], np.array([[fx, 0, cx], [0, fy, cy], [0, 0, 1]]), num_levels=c["levels"])
    return {"tracker": tr, "image": torch.from_numpy(_gray(frame)).cuda(),
            "depth": torch.from_numpy(_fine_depth(frame, seed)).cuda(),
            "levels": [[tr.level_buffer(l, q).torch() for q in range(6)] for l in range(c["levels"])]}


def _run_pyramids(s):
    s["tracker"].SetTrackingImage(s["image"])
    s["tracker"].SetTrackingDepth(s["depth"])
    return s["levels"]


def _exact_pyramids(c, seed):
    frame = _scene(seed).render(0, c["w"], c["h"])
    image = _gray(frame).astype(np.float64)
    z = _fine_depth(frame, seed)
    ok = (z > np.float32(0.2)) & (z < np.float32(8.0))
    inv = np.where(ok, 1.0 / np.where(ok, z, 1).astype(np.float64), 0.0)
    out = []
    for l in range(c["levels"]):
        fx, fy, cx, cy = (v / (1 << l) for v in synth.intrinsics(c["w"], c["h"]))
        if l:
            h, w = c["h"] >> l, c["w"] >> l
            k = np.array([1, 4, 6, 4, 1]) / 16.0
            at = [np.abs(2 * np.arange(n)[:, None] + np.arange(-2, 3)) for n in (h, w)]
            at = [np.where(a >= m, 2 * (m - 1) - a, a) for a, m in zip(at, image.shape)]
            image = np.einsum("yi,yixj,xj->yx", np.broadcast_to(k, at[0].shape),
                              image[at[0][:, :, None, None], at[1][None, None]], np.broadcast_to(k, at[1].shape))
            inv = inv[:2 * h:2, :2 * w:2].copy()
            inv[-1, :] = 0
            inv[:, -1] = 0
        h, w = image.shape
        gx, gy = np.zeros((h, w)), np.zeros((h, w))
        gx[1:-1, 1:-1] = (image[1:-1, 2:] - image[1:-1, :-2]) * 0.5
        gy[1:-1, 1:-1] = (image[2:, 1:-1] - image[:-2, 1:-1]) * 0.5
        zz = 1.0 / np.where(inv > 0, inv, 1)
        seen = (inv > 0) & (zz < 3.0)
        y, x = np.mgrid[:h, :w]
        v = np.stack([zz * (x - cx) / fx, zz * (y - cy) / fy, zz, np.ones((h, w))], -1)
        v = np.where(seen[..., None], v, np.array([0, 0, 0, -1.0]))
        nrm = np.zeros((h, w, 4))
        nrm[..., 3] = -1
        both = seen[:-1, :-1] & seen[:-1, 1:] & seen[1:, :-1]
        n = np.cross(v[1:, :-1, :3] - v[:-1, :-1, :3], v[:-1, 1:, :3] - v[:-1, :-1, :3])
        n /= np.maximum(np.linalg.norm(n, axis=-1, keepdims=True), 1e-300)
        nrm[:-1, :-1] = np.where(both[..., None], np.concatenate([n, np.ones(n.shape[:2] + (1,))], -1), nrm[:-1, :-1])
        out.append([image, gx, gy, inv, v, nrm])
    return out


# ---------------------------------------------------------------- mesh
def _saved_in_order(m, path):
    """Saves the map with its blocks in coordinate order (the pool's own order
    is that of their allocation, which no two runs share)."""
    m.SaveToFile(path)
    raw = np.fromfile(path, dtype=np.uint8)
    n = int(raw[44:48].view(np.uint32)[0])
    xyz = raw[144:144 + 12 * n].view(np.int32).reshape(n, 3)
    vox = raw[144 + 12 * n:].reshape(n, -1)
    order = np.lexsort((xyz[:, 0], xyz[:, 1], xyz[:, 2]))
    with open(path, "wb") as f:
        f.write(raw[:144].tobytes())
        f.write(xyz[order].tobytes())
        f.write(vox[order].tobytes())


def _prepare_mesh_view(c, seed):
    frames, poses = _frames(seed, c["frames"], c["w"], c["h"])
    K = synth.intrinsics(c["w"], c["h"])
    built = _map(K, c["vs"], c["fmt"])
    for f, T in zip(frames, poses):
        built.Fuse(_metres(f), T)
    with tempfile.TemporaryDirectory() as folder:
        path = os.path.join(folder, "submap.yas")
        _saved_in_order(built, path)
        built.Release()
        m = _map(K, c["vs"], c["fmt"])
        m.ReadFromFile(path)
    Tcw = np.eye(4)
    Tcw[:3, 3] = (0.05, -0.03, 0.6)  # the viewer stands back from the submap
    return {"map": m, "mesher": rf.MeshEngine(MAX_TRIANGLES), "canvas": rf.Canvas(c["w"], c["h"], K), "Tcw": Tcw,
            "triangles": rf.C.c_uint(),
            # the program's own triangle soup, as the reference's callers keep one
            "points": np.zeros((MAX_TRIANGLES, 9), np.float32), "normals": np.zeros((MAX_TRIANGLES, 9), np.float32),
            "cases": np.zeros(MAX_TRIANGLES, np.int32), "cubes": np.zeros((MAX_TRIANGLES, 3), np.int32)}


def _run_mesh_view(s):
    mesher, call = s["mesher"].handle, rf.L.call
    call("yas_mesher_meshify", mesher, s["map"].handle, rf.C.byref(s["triangles"]))
    call("yas_mesher_copy", mesher, s["points"].ctypes.data, s["normals"].ctypes.data, MAX_TRIANGLES)
    call("yas_mesher_copy_cases", mesher, s["cases"].ctypes.data, s["cubes"].ctypes.data, MAX_TRIANGLES)
    s["canvas"].clear()
    s["canvas"].draw_mesh(s["mesher"], np.eye(4), s["Tcw"])
    rgba, depth = s["canvas"].read()
    return {"triangles": s["triangles"].value, "points": s["points"], "normals": s["normals"], "cases": s["cases"],
            "cubes": s["cubes"], "rgba": rgba, "depth": depth}


# ---------------------------------------------------------------- the interface
_PREPARE = {"session": _prepare_session, "batch": _prepare_batch, "served": _prepare_served,
            "fuse_raycast": _prepare_fuse_raycast, "reintegrate": _prepare_reintegrate, "track": _prepare_track,
            "pyramids": _prepare_pyramids, "mesh_view": _prepare_mesh_view}
_RUN = {"session": _run_session, "batch": _run_batch, "served": _run_served, "fuse_raycast": _run_fuse_raycast,
        "reintegrate": _run_reintegrate, "track": _run_track, "pyramids": _run_pyramids, "mesh_view": _run_mesh_view}


def prepare(case, seed):
    state = _PREPARE[case["use"]](case, int(seed))
    state["use"] = case["use"]
    return state


def run(state):
    return _RUN[state["use"]](state)


def exact(case, seed):
    # the pyramids have a closed form; a map, its raycast, its mesh and a track
    # are whole calls with per-sample decisions on single-precision values
    return _exact_pyramids(case, int(seed)) if case["use"] == "pyramids" else None


def _blocks(vs):
    """Blocks in view: about 21 m^2 of surface band at the scenes' sizes."""
    return 21.0 / (8 * vs) ** 2


def _pyramid_pixels(w, h, levels):
    return sum((w >> l) * (h >> l) for l in range(levels))


def _frame_work(w, h, vs, fmt):
    """A tracked and fused frame: input (5 B), pyramids written and read once
    (48 B current, 40 B reference per pixel and level), the blocks in view read
    and written by fusion and read by the raycast; the Gauss-Newton products."""
    p, px, vb = w * h, _pyramid_pixels(w, h, 3), 8 if fmt == "f32" else 4
    it = sum(n * (w >> l) * (h >> l) for l, n in enumerate(ITERATIONS[:3]))
    return {"bytes": 5 * p + 2 * 88 * px + 16 * p + 3 * 512 * vb * _blocks(vs), "flops": 300 * it + 60 * 512 * _blocks(vs)}


def work(case):
    use = case["use"]
    w, h = case.get("w", 0), case.get("h", 0)
    if use == "session":
        return _frame_work(w, h, case["vs"], case["fmt"])
    if use in ("batch", "served"):
        each = [_frame_work(a, b, case["vs"] if i % 2 or use == "served" else max(case["vs"], 0.008), case["fmt"])
                for i, (a, b) in enumerate(_sizes(case["n"]))]
        return {k: sum(e[k] for e in each) for k in ("bytes", "flops")}
    if use in ("track", "pyramids"):
        px = _pyramid_pixels(w, h, case["levels"])
        if use == "pyramids":
            return {"bytes": 5 * w * h + 48 * px, "flops": 60 * px}
        it = sum(n * (w >> l) * (h >> l) for l, n in enumerate(ITERATIONS[:case["levels"]]))
        return {"bytes": 5 * w * h + 48 * px + 88 * px, "flops": 300 * it}
    vb = 8 if case["fmt"] == "f32" else 4
    blocks = _blocks(case["vs"])
    if use == "fuse_raycast":
        return {"bytes": 20 * w * h + 3 * 512 * vb * blocks, "flops": 60 * 512 * blocks}
    if use == "reintegrate":
        n = case["frames"]
        return {"bytes": n * (8 * w * h + 4 * 512 * vb * blocks) + 16 * w * h + 512 * vb * blocks,
                "flops": 120 * n * 512 * blocks}
    triangles = 90 * blocks
    return {"bytes": 512 * vb * blocks + 2 * 88 * triangles + 8 * w * h, "flops": 200 * triangles}
