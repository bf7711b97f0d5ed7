"""Device memory that a context takes for paths it does not run.

The second set of per-face measurements belongs to pipelined steps, which a
bulk-modulus context does not make; the split records and face-wise patch ids
belong to element kernels that an FP64 SMOOTH context runs only when told to (and
then gets them).  Level 7, so that each table exceeds the allocator's 2 MB."""
import numpy as np
import pytest

from shell_gb300 import lib as L
from tests.common import physics_params

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_bulk_modulus_has_no_second_set(cuda_ok):
    X, T = L.icosphere(7)
    L.Shell(X, T, physics_params(contact=False)).close()  # what the first context leaves behind
    took = []
    for bulk in (0.0, 1e-3):
        before = _free()
        g = L.Shell(X, T, physics_params(contact=False, bulk_modulus=bulk))
        took.append(before - _free())
        g.close()
    assert took[0] - took[1] >= 5 * 8 * len(T) - 5 * 2 * MB


def test_split_records_of_a_smooth_context_on_demand(cuda_ok):
    X, T = L.icosphere(6)
    g = L.Shell(X, T, physics_params(shell_shell_contact=L.CONTACT_SMOOTH))
    u = 1e-3 * np.random.default_rng(0).standard_normal(X.size)
    z = np.zeros_like(u)
    f0 = g.eval_forces(u, z, -1e-4)[0]
    before = _free()
    g.set_element_variant(6)
    assert before - _free() >= (416 + 48) * len(T) - 2 * 2 * MB
    f1 = g.eval_forces(u, z, -1e-4)[0]
    assert np.linalg.norm(f1 - f0) / np.linalg.norm(f0) < 1e-12
    g.set_element_variant(-1)
    assert np.array_equal(g.eval_forces(u, z, -1e-4)[0].view(np.uint64), f0.view(np.uint64))
    g.close()
