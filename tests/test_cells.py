"""The cells that a face's box covers (shl_cells.h) against the three loops over
them: every extent of one to a few cells, and ranges empty on one axis or more,
down to those of a box without a node (INT_MAX to INT_MIN), which cover none.
Compiled from the header the kernels use."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r'''
#include "shl_cells.h"
extern "C" unsigned covered(const int* lo, const int* hi) { return shl_cells_covered(lo, hi); }
extern "C" unsigned at(unsigned q, const int* lo, const int* hi, unsigned ny, unsigned nz) {
  return shl_cells_at(q, lo, hi, ny, nz);
}
'''


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("cells")
    (d / "h.cpp").write_text(HARNESS)
    so = d / "libh.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", os.path.join(ROOT, "shell_gb300", "csrc"),
                    str(d / "h.cpp"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.covered.restype = lib.at.restype = ctypes.c_uint
    lib.covered.argtypes = [ctypes.c_void_p] * 2
    lib.at.argtypes = [ctypes.c_uint, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint, ctypes.c_uint]
    return lib


def _cells(lib, lo, hi, ny, nz):
    lo, hi = np.array(lo, dtype=np.int32), np.array(hi, dtype=np.int32)
    n = lib.covered(lo.ctypes.data, hi.ctypes.data)
    return n, [lib.at(q, lo.ctypes.data, hi.ctypes.data, ny, nz) for q in range(min(n, 1000))]


def test_same_cells_as_the_loops(harness):
    rng = np.random.default_rng(0)
    for _ in range(2000):
        ny, nz = (int(x) for x in rng.integers(1, 40, 2))
        lo = [int(rng.integers(0, 9)), int(rng.integers(0, ny)), int(rng.integers(0, nz))]
        hi = [lo[0] + int(rng.integers(-2, 5)), int(rng.integers(max(lo[1] - 2, 0), min(lo[1] + 5, ny))),
              int(rng.integers(max(lo[2] - 2, 0), min(lo[2] + 5, nz)))]
        want = [x * ny * nz + y * nz + z for x in range(lo[0], hi[0] + 1) for y in range(lo[1], hi[1] + 1)
                for z in range(lo[2], hi[2] + 1)]
        assert _cells(harness, lo, hi, ny, nz) == (len(want), want)


@pytest.mark.parametrize("axes", [(0,), (1,), (2,), (0, 1), (0, 2), (1, 2), (0, 1, 2)])
def test_box_without_a_node_covers_none(harness, axes):
    lo, hi = [3, 4, 5], [4, 4, 6]
    for c in axes:
        lo[c], hi[c] = 2 ** 31 - 1, -2 ** 31
    assert _cells(harness, lo, hi, 20, 20) == (0, [])
