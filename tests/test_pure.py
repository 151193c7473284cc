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
extern "C" size_t image_bytes(size_t row, size_t pitch, int rows) { return yas::image_bytes(row, pitch, rows); }
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
