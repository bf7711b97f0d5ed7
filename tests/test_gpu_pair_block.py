"""The block-wide pruned closest-point search (shl_pairs.cuh) against the fifteen
tests in a row, both on the device, bit for bit.

The device build of the bounds (FP32 contraction, fast division, rsqrt) and the
dealing out of the tests over a block are not those of the host build, so the
kinds of pairs of the host test pass through them here: several trips of each
block and a partly filled last one.  NaN of either sign, too: a NaN keeps out of
the minimum whatever its bits.  The largest miss of the FP32 edge-edge distance
on these pairs stays below the margin that the bounds allow for it."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from shell_gb300 import build
from tests.test_pair_prune import pairs

pytestmark = pytest.mark.gpu

HARNESS = r'''
#include <cuda_runtime.h>
#include "shl_pairs.cuh"
using namespace shl;
// p: n x 6 x 3 doubles; out: n x 8 doubles (d2, dc, v, w)
__device__ void put(double* o, const shl_pair_geom& g) {
  o[0] = g.d2; o[1] = g.dc[0]; o[2] = g.dc[1]; o[3] = g.dc[2];
  o[4] = g.v[0]; o[5] = g.v[1]; o[6] = g.w[0]; o[7] = g.w[1];
}
__global__ void __launch_bounds__(kPairBlock) k_block(const double* p, unsigned n, double* out) {
  extern __shared__ __align__(16) unsigned char smem[];
  PairWork& work = *reinterpret_cast<PairWork*>(smem);
  for (unsigned j0 = blockIdx.x * blockDim.x; j0 < n; j0 += gridDim.x * blockDim.x) {
    const unsigned j = j0 + threadIdx.x;
    const bool active = j < n;
    const double* q = p + 18 * (size_t)(active ? j : j0);
    const double* a[3] = {q, q + 3, q + 6};
    const double* b[3] = {q + 9, q + 12, q + 15};
    shl_pair_geom g;
    pair_compute_block(active, a, b, work, &g);
    if (active) put(out + 8 * (size_t)j, g);
  }
}
// miss: bits of the largest |FP32 - FP64| edge-edge squared distance, in the bounds' unit length
__global__ void k_full(const double* p, unsigned n, double* out, unsigned* miss) {
  const unsigned j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const double* q = p + 18 * (size_t)j;
  const double* a[3] = {q, q + 3, q + 6};
  const double* b[3] = {q + 9, q + 12, q + 15};
  shl_pair_geom g;
  shl_pair_compute(a, b, &g);
  put(out + 8 * (size_t)j, g);
  float P[6][3], M2 = 0.f;
  for (int k = 0; k < 6; ++k) {
    for (int c = 0; c < 3; ++c) P[k][c] = (float)SHL_SUB(q[3 * k + c], q[c]);
    M2 = fmaxf(M2, shl_f3_dot(P[k], P[k]));
  }
  if (!(M2 > 1e-30f && M2 < 1e30f)) return;
  const float sc = SHL_RSQRTF(M2);
  for (int k = 0; k < 6; ++k)
    for (int c = 0; c < 3; ++c) P[k][c] *= sc;
  for (int i = 0; i < 3; ++i)
    for (int m = 0; m < 3; ++m) {
      float d1[3], d2[3], r[3];
      for (int c = 0; c < 3; ++c) {
        d1[c] = P[(i + 1) % 3][c] - P[i][c];
        d2[c] = P[3 + (m + 1) % 3][c] - P[3 + m][c];
        r[c] = P[i][c] - P[3 + m][c];
      }
      const float x = shl_f_segments(d1, d2, r, shl_f3_dot(d1, d1), shl_f3_dot(d2, d2));
      double dc[3], st[2];
      shl_segment_segment(a[i], a[(i + 1) % 3], b[m], b[(m + 1) % 3], dc, st);
      const double y = shl_v3_dot(dc, dc) * (double)sc * (double)sc;
      const float e = (float)fabs((double)x - y);
      if (e == e) atomicMax(miss, __float_as_uint(e));
    }
}
extern "C" int run(const double* p, unsigned n, double* block, double* full, float* miss) {
  double *dp, *db, *df;
  unsigned* dm;
  int e = cudaMalloc(&dp, 18 * sizeof(double) * n) || cudaMalloc(&db, 8 * sizeof(double) * n) ||
          cudaMalloc(&df, 8 * sizeof(double) * n) || cudaMalloc(&dm, 4);
  e = e || cudaMemcpy(dp, p, 18 * sizeof(double) * n, cudaMemcpyHostToDevice) || cudaMemset(dm, 0, 4);
  e = e || cudaFuncSetAttribute((const void*)k_block, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(PairWork));
  if (!e) {
    k_block<<<100, kPairBlock, sizeof(PairWork)>>>(dp, n, db);
    k_full<<<(n + 127) / 128, 128>>>(dp, n, df, dm);
    e = cudaMemcpy(block, db, 8 * sizeof(double) * n, cudaMemcpyDeviceToHost) ||
        cudaMemcpy(full, df, 8 * sizeof(double) * n, cudaMemcpyDeviceToHost) ||
        cudaMemcpy(miss, dm, 4, cudaMemcpyDeviceToHost);
  }
  cudaFree(dp); cudaFree(db); cudaFree(df); cudaFree(dm);
  return e;
}
'''


@pytest.fixture(scope="module")
def harness(cuda_ok, tmp_path_factory):
    d = tmp_path_factory.mktemp("pairs")
    (d / "h.cu").write_text(HARNESS)
    so = d / "libh.so"
    subprocess.run([build.NVCC] + build.NVCC_FLAGS + ["-I", build.CSRC, "-shared", str(d / "h.cu"), "-o", str(so)],
                   check=True)
    lib = ctypes.CDLL(str(so))
    lib.run.argtypes = [ctypes.c_void_p, ctypes.c_uint, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
    return lib


@pytest.mark.parametrize("kind", ["general", "layers", "stacked", "parallel", "slivers", "touching", "grid", "flat",
                                  "degenerate", "far", "scales", "nonfinite", "signed nan"])
def test_block_search_equals_full(harness, kind):
    n = 100037
    rng = np.random.default_rng(5)
    p = pairs("nonfinite" if kind == "signed nan" else kind, n, rng)
    if kind == "signed nan":
        p[np.isnan(p)] = np.copysign(np.nan, -1.0)
        p[n // 2:] = np.where(np.isinf(p[n // 2:]), np.copysign(np.nan, -1.0), p[n // 2:])
    block, full = np.zeros((n, 8)), np.zeros((n, 8))
    miss = np.zeros(1, dtype=np.float32)
    assert harness.run(p.ctypes.data, n, block.ctypes.data, full.ctypes.data, miss.ctypes.data) == 0
    assert np.array_equal(block.view(np.uint64), full.view(np.uint64))
    print("%s: edge-edge miss %.1f eps" % (kind, miss[0] / 2.0 ** -24))
    assert miss[0] <= 128 * 2.0 ** -24
