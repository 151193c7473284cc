"""The fused Gauss-Newton schedule where its variants and its arithmetic change.

It finds a pixel's row with a multiplication, projects the model through an
approximate reciprocal (the exact form only near a pixel's edge), gates on
squares, and is compiled for 1, 2, 4 or any number of pixels per thread and for
the RGBD mode alone.  Against the per-iteration kernels, which do none of this:
one iteration's normal equations agree within 1e-5 of the largest entry (both
sum the same products, at most some tens of FP32 additions of 2^-24 each before
the compensated sums; a pixel gained or lost in the small images is above it),
and the pose of a schedule within the 2e-5 m / rad of the other schedule tests.
Sizes: the smallest level (4 x 4), less than a warp's row, ragged, and one on
each side of every pixels-per-thread step.
A batch of one mode runs the same code as one of several: equal bits.
"""
from __future__ import annotations

import numpy as np
import pytest

from tests.helpers import pose_error, sequence
from yetanotherslam_gb300 import batching, synth
from yetanotherslam_gb300 import rgbdfusion as rf

pytestmark = pytest.mark.gpu

SIZES = [(4, 4, 1), (37, 23, 2), (333, 251, 3), (319, 241, 1), (480, 320, 2), (641, 480, 1), (1279, 721, 3)]


def _tracker(mode, w, h, levels, iters):
    fx, fy, cx, cy = synth.intrinsics(w, h)
    K = np.array([[fx, 0, cx], [0, fy, cy], [0, 0, 1.0]])
    seq = sequence(11, 2, w, h)
    tr = rf.RGBDTracking(w, h, K, bRGB=bool(mode & 1), bIcp=bool(mode & 2), num_levels=levels, iterations=iters)
    tr.SetReferenceImage(synth.gray_of(seq[0][0]))
    tr.SetReferenceDepth(seq[0][2])
    tr.SetTrackingImage(synth.gray_of(seq[1][0]))
    tr.SetTrackingDepth(seq[1][2])
    m = rf.MapStruct(K)
    m.create_config(1 << 18, 1 << 16, 0.008, 0.024, rf.VOXEL_F32)
    m.Fuse(seq[0][2], np.eye(4))
    rc = rf.RayTraceEngine(w, h, K)
    rc.RayTrace(m, np.eye(4))
    tr.SetReferenceModel(rc.GetVMap())
    return tr


@pytest.mark.parametrize("mode", [1, 2, 3])
@pytest.mark.parametrize("w,h,levels", SIZES)
def test_one_iteration_matches_the_per_iteration_kernels(cuda, w, h, levels, mode):
    init = np.eye(4)
    init[:3, 3] = [0.004, -0.002, 0.003]
    for level in range(levels):
        tr = _tracker(mode, w, h, levels, [int(l == level) for l in range(levels)])
        out = []
        for fused in (True, False):
            tr.set_schedule(fused)
            T = tr.GetTransform(init, False)
            out.append((T, tr.last_solve()[0]))
        (Tf, Hf), (Tp, Hp) = out
        assert np.abs(Hf - Hp).max() <= 1e-5 * np.abs(Hp).max(), level
        if np.linalg.cond(Hp) < 1e6:
            dt, dr = pose_error(Tp, Tf)
            assert dt <= 2e-5 and dr <= 2e-5, (level, dt, dr)


def test_modes_mixed_in_a_batch_match_each_mode_alone(cuda):
    tuning = batching.default_tuning()
    tuning.gn_pixels_per_cta = 32768

    def run(modes):
        ss = [rf.Session(w, h, synth.intrinsics(w, h), mode=mode) for w, h, mode in modes]
        b = batching.Batch(ss)
        b.tuning = tuning
        seqs = [sequence(3, 4, w, h) for w, h, _ in modes]
        out = []
        for f in range(4):
            b.step([(q[f][0], q[f][1]) for q in seqs])
            P, st, _ = b.wait()
            assert not np.any(st)
            out.append(np.array(P))
        return np.array(out)

    items = [(161, 119, 1), (320, 240, 2), (251, 187, 3), (64, 48, 2)]
    mixed = run(items)
    for i, it in enumerate(items):
        assert np.array_equal(mixed[:, i], run([it])[:, 0]), it
