"""The pruned closest-point search of a triangle pair against the full one.

shl_pair_mask (shl_prune.h) bounds the fifteen tests of a pair in FP32 and
drops those that cannot hold the minimum; shl_pair_compute_masked over the rest
must give shl_pair_compute's result bit for bit, for every kind of pair: in
general position, stacked in layers, with parallel, coincident, touching,
collinear or zero edges, slivers and needles, coordinates on a grid, flat or far
from the origin, at any scale, and with infinities and NaN (every test kept).
Compiled from the headers the kernels use (g++, -ffp-contract=off).
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HARNESS = r'''
#include <string.h>
#include "shl_geom.h"
#include "shl_prune.h"
// pairs: n x 6 x 3 doubles; returns the number of differing results, *tests the tests kept
extern "C" long compare(const double* p, long n, long* tests) {
  long bad = 0;
  *tests = 0;
  for (long i = 0; i < n; ++i, p += 18) {
    const double* a[3] = {p, p + 3, p + 6};
    const double* b[3] = {p + 9, p + 12, p + 15};
    shl_pair_geom g, h;
    memset(&g, 0, sizeof g);
    memset(&h, 0, sizeof h);
    shl_pair_compute(a, b, &g);
    const unsigned m = shl_pair_mask(a, b);
    shl_pair_compute_masked(a, b, m, &h);
    *tests += __builtin_popcount(m);
    if (memcmp(&g, &h, sizeof g)) ++bad;
  }
  return bad;
}
'''


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("prune")
    (d / "h.cpp").write_text(HARNESS)
    so = d / "libh.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-ffp-contract=off",
                    "-I", os.path.join(ROOT, "shell_gb300", "csrc"), str(d / "h.cpp"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.compare.restype = ctypes.c_long
    lib.compare.argtypes = [ctypes.c_void_p, ctypes.c_long, ctypes.POINTER(ctypes.c_long)]
    return lib


def pairs(kind, n, rng):
    p = rng.standard_normal((n, 6, 3))
    gap = 10.0 ** (-7 * rng.random((n, 1)))
    fine = 10.0 ** (-8 * rng.random((n, 1)))
    t = rng.random((n, 1))
    if kind == "layers":
        p[:, :, 2] = 1e-9 * rng.standard_normal((n, 6))
        p[:, 3:, 2] += gap
    elif kind == "stacked":
        p[:, 3:] = p[:, :3] + 1e-8 * gap[:, None] * rng.standard_normal((n, 3, 3))
        p[:, 3:, 2] += gap
    elif kind == "parallel":
        p[:, 4] = p[:, 3] + (p[:, 1] - p[:, 0]) * (1 + 0.1 * rng.standard_normal((n, 1))) + fine * rng.standard_normal((n, 3))
    elif kind == "slivers":
        p[:, 2] = p[:, 0] * (1 - t) + p[:, 1] * t + fine * rng.standard_normal((n, 3))
        p[:, 5] = p[:, 4] + fine * rng.standard_normal((n, 3))
    elif kind == "touching":
        p[:, 3] = p[:, 0] + gap * rng.standard_normal((n, 3))
    elif kind == "grid":
        p = np.round(2 * p)
        p[:, 3:, 2] += np.where(rng.random((n, 1)) < 0.5, gap, 0.0)
    elif kind == "flat":
        p *= np.array([1.0, 10.0 ** -2.5, 1e-4])
        p[:, 3:, 2] += gap
    elif kind == "degenerate":
        p[:, 1] = p[:, 0]
        p[::2, 2] = p[::2, 0]
        p[::3, 4] = p[::3, 5]
    elif kind == "far":
        p *= 10.0 ** (-2.5 * rng.random((n, 1, 1)))
        p[:, :, 0] += 10.0 ** (3 * rng.random((n, 1)))
        p[:, 3:, 2] += gap
    elif kind == "scales":
        p *= 10.0 ** rng.uniform(-120, 120, (n, 1, 1))
    elif kind == "nonfinite":
        p[np.arange(n), rng.integers(0, 6, n), rng.integers(0, 3, n)] = rng.choice([np.nan, np.inf, -np.inf, 1e300], n)
    return np.ascontiguousarray(p)


@pytest.mark.parametrize("kind", ["general", "layers", "stacked", "parallel", "slivers", "touching", "grid", "flat",
                                  "degenerate", "far", "scales", "nonfinite"])
def test_pruned_equals_full(harness, kind):
    n = 100000
    p = pairs(kind, n, np.random.default_rng(5))
    kept = ctypes.c_long()
    assert harness.compare(p.ctypes.data, n, ctypes.byref(kept)) == 0
    if kind == "general":
        assert kept.value < 5 * n  # the bounds do prune: 1.9 of 15 tests on random pairs
