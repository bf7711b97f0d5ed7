"""A residual whose device buffers do not all fit, and the same call once they do.

The library's own sources, linked with an allocator that fails at the k-th
request, for every request that a first FP64 residual of an FP32 context makes.
The call reports the lack of memory; repeated with memory to be had, it gives the
residual, and the steps after it the state, of a context that never failed."""
import os
import subprocess

import numpy as np
import pytest

from shell_gb300 import build, lib as L
from tests.common import cell_size_mult_for, physics_params

pytestmark = pytest.mark.gpu

ALLOCATOR = r'''
#include <cuda_runtime.h>
static int fail_at = 0, requests = 0;
extern "C" cudaError_t shl_test_malloc(void** p, size_t n) {
  ++requests;
  if (fail_at > 0 && --fail_at == 0) return cudaErrorMemoryAllocation;
  return cudaMalloc(p, n);
}
extern "C" void shl_test_fail(int k) { fail_at = k; requests = 0; }
extern "C" int shl_test_requests(void) { return requests; }
'''


@pytest.fixture(scope="module")
def library(cuda_ok, tmp_path_factory):
    d = tmp_path_factory.mktemp("alloc")
    (d / "a.cu").write_text(ALLOCATOR)
    api = str(d / "api.o")
    jobs = [subprocess.Popen([build.NVCC] + build.NVCC_FLAGS + args) for args in (
        ["-DcudaMalloc=shl_test_malloc", "-c", os.path.join(build.CSRC, "shl_api.cu"), "-o", api],
        ["-c", str(d / "a.cu"), "-o", str(d / "a.o")])]
    assert [j.wait() for j in jobs] == [0, 0]
    rest = [os.path.join(build.OUT, s + ".o") for s in build.CU_SOURCES + build.CPP_SOURCES if s != "shl_api.cu"]
    so = str(d / "libshl_test.so")
    subprocess.run([build.NVCC] + build.ARCH + ["-shared", "-o", so, api, str(d / "a.o")] + rest +
                   ["-Xcompiler", "-fopenmp", "-lgomp"], check=True)
    return so


@pytest.mark.parametrize("contact", [L.CONTACT_NONE, L.CONTACT_SMOOTH])
def test_residual_after_a_failed_allocation(library, monkeypatch, contact):
    monkeypatch.setattr(L, "LIB_PATH", library)
    monkeypatch.setattr(L, "_lib", None)
    lib = L.load()
    X, T = L.icosphere(2)
    p = physics_params(shell_shell_contact=contact, precision=L.PREC_FP32, cell_size_mult=cell_size_mult_for(X, T, 0.01))
    u = 1e-3 * np.random.default_rng(4).standard_normal(X.size)
    flags = L.RESIDUAL_FP64 | L.RESIDUAL_CORRECT

    def run(k):
        g = L.Shell(X, T, p)
        g.set_state(u, np.zeros_like(u), np.zeros_like(u))
        lib.shl_test_fail(k)
        if k:
            with pytest.raises(L.ShlError, match="103"):
                g.residual(-1e-5, flags)
            lib.shl_test_fail(0)
        r = g.residual(-1e-5, flags)
        n = lib.shl_test_requests()
        g.step(3, np.full(3, -1e-5))
        out = [r] + list(g.get_state())
        g.close()
        return n, [np.ascontiguousarray(x).view(np.uint64) for x in out]

    n, want = run(0)
    assert n >= 6
    for k in range(1, n + 1):
        for x, y in zip(run(k)[1], want):
            assert np.array_equal(x, y), k
