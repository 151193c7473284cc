"""The arithmetic of csrc/pure.h, compiled for the host."""
from __future__ import annotations

import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "yetanotherslam_gb300" / "csrc"
HARNESS = """
#include "pure.h"
#include <cstdint>

// Cells whose blocks' pool indices are drawn around the grid's limit, corner by
// corner against the blocks they were drawn from; the cells that differ.
extern "C" int corner_mismatches(int cells, int inner) {
    const int64_t ask = yas::kGridAsk;
    uint64_t state = 88172645463325252ull;
    const auto next = [&] { state ^= state << 13; state ^= state >> 7; state ^= state << 17; return state; };
    int bad = 0;
    for (int n = 0; n < cells; ++n) {
        const unsigned across = 1u + (unsigned)(next() % 7);
        int block[8];
        for (int d = 0; d < 8; ++d) {
            const int64_t near_limit = ask - 3 + (int64_t)(next() % 6), small = (int64_t)(next() % 1000);
            const uint64_t kind = next() % 8;
            block[d] = (int)(kind < 3 ? small : kind < 6 ? near_limit : kind == 6 ? 0x7fffffff : -1);
        }
        if (block[0] < 0) block[0] = 5;  // the block that holds corner 0 is allocated
        unsigned q[8];
        const auto word = [&](unsigned c) {
            const int e = block[c & across];
            return e < 0 ? 0x1000000u + (unsigned)(next() % 0xfe000000u) : e < ask ? (unsigned)e : yas::kGridAsk;
        };
        const unsigned lim = yas::corner_blocks(across, block[0], inner != 0, word, [&](unsigned d) { return block[d]; }, q);
        bool same = true;
        for (unsigned c = 0; c < 8; ++c) same = same && (q[c] < lim ? (int)q[c] : -1) == block[c & across];
        bad += same ? 0 : 1;
    }
    return bad;
}

extern "C" size_t image_bytes(size_t row, size_t pitch, int rows) { return yas::image_bytes(row, pitch, rows); }
extern "C" void huber_scaled(const float *sd, float *out, int n) {
    for (int i = 0; i < n; ++i) out[i] = yas::huber_scaled(sd[i]);
}
"""


@pytest.fixture(scope="module")
def pure(tmp_path_factory):
    d = tmp_path_factory.mktemp("pure")
    (d / "pure.cpp").write_text(HARNESS)
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-ffp-contract=off", "-fPIC", "-shared",
                        f"-I{CSRC}", str(d / "pure.cpp"), "-o", str(d / "libpure.so")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return C.CDLL(str(d / "libpure.so"))


@pytest.mark.parametrize("w,h,pad", [(1, 1, 0), (1, 1, 15), (37, 23, 0), (37, 23, 3), (640, 480, 128), (5, 1, 11)])
def test_an_image_ends_with_its_last_rows_own_bytes(pure, w, h, pad):
    pure.image_bytes.restype = C.c_size_t
    a = np.zeros((h, w + pad), np.float32)
    view = a[:, :w]  # numpy's own idea of where a padded image ends
    first, last = np.lib.array_utils.byte_bounds(view)
    assert pure.image_bytes(C.c_size_t(4 * w), C.c_size_t(4 * (w + pad)), h) == last - first


@pytest.mark.parametrize("inner", [0, 1])
def test_corner_blocks_at_the_grids_index_limit(pure, inner):
    assert pure.corner_mismatches(200000, inner) == 0


def test_huber_scale_rounds_once(pure):
    """Every deviation of two binades, and the ends of the range."""
    sd = np.concatenate([np.arange(0x3f800000, 0x40800000, dtype=np.uint32).view(np.float32),
                         np.array([0, 1e-45, 1e-38, 7e37, 3.4e38, np.inf, np.nan], np.float32)])
    out = np.empty_like(sd)
    pure.huber_scaled(sd.ctypes.data_as(C.c_void_p), out.ctypes.data_as(C.c_void_p), sd.size)
    with np.errstate(over="ignore"):
        want = (4.685 * sd.astype(np.float64)).astype(np.float32)
    assert np.array_equal(out.view(np.uint32)[:-1], want.view(np.uint32)[:-1]) and np.isnan(out[-1])
