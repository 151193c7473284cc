"""Values of every voxel format after frames are fused, and after the last is removed
again, against the oracle's FP32 maps of the same frames.

Bounds, in units of the truncation.  The kernel's FP32 arithmetic: the new sample is
a product with a rounded reciprocal where the oracle divides (3 x 2^-24), an update a
fused sum times an approximate reciprocal (3 x 2^-24) where the oracle rounds three
times: under 7.2e-7 a frame, 2e-6 for three.  A word's own rounding r (F16 2^-20: 18
bits of a value below 1; S24 2^-23; S16 truncates, 1/32767; F32 none) adds r to a
first write, 1/2 r + r to a second, 2/3 (3/2 r) + r = 2 r to a third.  Removing a
frame multiplies a voxel's error by w / (w - 1), at most 2 (of 3/2 r) or 3/2 (of 2 r),
and rounds once more: 4 r, and 2 x 2e-6.
"""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from tests.helpers import align_blocks, key_rows
from tests.test_gpu_integrate import CASES
from yetanotherslam_gb300 import rgbdfusion as rf

pytestmark = pytest.mark.gpu

ROUNDING = {"f32": 0.0, "f16": 2.0 ** -20, "s24": 2.0 ** -23, "s16": 1.0 / 32767}
FORMAT = {"f32": rf.VOXEL_F32, "f16": rf.VOXEL_F16, "s24": rf.VOXEL_S24, "s16": rf.VOXEL_S16}


@pytest.mark.parametrize("w,h,fx,fy,cx,cy", CASES)
@pytest.mark.parametrize("fmt", sorted(ROUNDING))
def test_fused_and_removed_values_match_oracle(cuda, w, h, fx, fy, cx, cy, fmt):
    rng = np.random.default_rng(w)
    K, r = (fx, fy, cx, cy), ROUNDING[fmt]
    m = rf.MapStruct(K)
    m.create_config(1 << 18, 1 << 15, 0.008, 0.024, FORMAT[fmt])
    two, three = oracle.Map(0.008, 0.024), oracle.Map(0.008, 0.024)
    T = np.eye(4)
    for k in range(3):
        d = rng.uniform(0.5, 0.9, (h, w)).astype(np.float32)
        d[rng.random((h, w)) < 0.1] = 0.0
        T[:3, 3] = rng.uniform(-0.02, 0.02, 3)
        m.Fuse(d, T)
        three.fuse(d, K, T)
        if k < 2:
            two.fuse(d, K, T)
    sa, wa, so, wo = align_blocks(*m.export(), *three.export())
    assert np.array_equal(wa, wo) and (w == 1 or (wo > 0).any())  # one pixel's voxels are all missed
    assert np.abs(sa - so)[wo > 0].max(initial=0.0) <= 2e-6 + 2 * r
    m.Defuse(d, T)
    cd, sd, wd = m.export()
    ct, st, wt = two.export()
    kd, kt = key_rows(cd), key_rows(ct)
    old = np.isin(kd, kt)  # blocks of the removed frame alone are empty
    assert not wd[~old].any()
    by, of = np.argsort(kd[old]), np.argsort(kt)
    assert np.array_equal(wd[old][by], wt[of])
    assert np.abs(sd[old][by] - st[of])[wt[of] > 0].max(initial=0.0) <= 4e-6 + 4 * r
