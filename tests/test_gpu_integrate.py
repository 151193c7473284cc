"""Depth integration where its pixel projection can go wrong.

The kernel projects through an approximate reciprocal and evaluates the
canonical quotient only near a pixel's edge, in images whose size and
principal point bound the difference (below 2^18 pixels); beyond, everywhere.
Against the oracle: block set and weights equal (the same voxels project into
the same valid pixels), TSDF within 1e-5 (the bound of the other fusion
tests).  Cases: one pixel, ragged sizes, a principal point outside the image,
and one so far out that every coordinate is evaluated exactly; frames fused
and removed again.
"""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from tests.helpers import align_blocks, key_rows
from yetanotherslam_gb300 import rgbdfusion as rf

pytestmark = pytest.mark.gpu

CASES = [  # width, height, fx, fy, cx, cy
    (1, 1, 40.0, 40.0, 0.0, 0.0),
    (37, 23, 45.0, 44.0, 18.2, 10.9),
    (130, 97, 160.0, 158.0, -41.5, 131.0),
    (2999, 61, 5.0e4, 120.0, 2.7e5, 30.0),
]


@pytest.mark.parametrize("w,h,fx,fy,cx,cy", CASES)
@pytest.mark.parametrize("fmt", [rf.VOXEL_F32, rf.VOXEL_F16])
def test_projection_edges_match_oracle(cuda, w, h, fx, fy, cx, cy, fmt):
    rng = np.random.default_rng(w)
    K = (fx, fy, cx, cy)
    m = rf.MapStruct(K)
    m.create_config(1 << 18, 1 << 15, 0.008, 0.024, fmt)
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
    cg, sg, wg = m.export()
    co, so, wo = three.export()
    assert len(cg) > 0 and m.take_errors() == 0
    sa, wa, so, wo = align_blocks(cg, sg, wg, co, so, wo)
    assert np.array_equal(wa, wo)
    assert np.abs(sa - so)[wo > 0].max(initial=0.0) <= (1e-5 if fmt == rf.VOXEL_F32 else 1e-3)
    m.Defuse(d, T)  # the weights of the first two frames again; the last one's own blocks are empty
    cd, sd, wd = m.export()
    ct, st, wt = two.export()
    kd, kt = key_rows(cd), key_rows(ct)
    old = np.isin(kd, kt)
    assert not wd[~old].any()
    assert np.array_equal(wd[old][np.argsort(kd[old])], wt[np.argsort(kt)])
