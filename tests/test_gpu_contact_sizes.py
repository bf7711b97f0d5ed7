"""The contact CSR's register sort at every size of its networks.

A node's entries are sorted by one warp in registers, in a network of 32, 64,
..., 1024 elements chosen by their number.  Squashed shells of several sizes,
gaps and modes have nodes in every one of these ranges (checked); two contexts
built from one state must give the same forces bit for bit, and an entry out of
order would carry the scatter's atomics' order into the sums."""
import numpy as np
import pytest

from shell_gb300 import lib as L
from shell_gb300.workloads import squashed_state, workload

pytestmark = pytest.mark.gpu

SEEN = set()


@pytest.mark.parametrize("level,contact,part", [(3, "linear", 1.0), (4, "linear", 1.0), (5, "linear", 0.3),
                                                (6, "linear", 1.0), (4, "smooth", 1.0), (5, "smooth", 0.6)])
def test_forces_do_not_depend_on_the_scatter(cuda_ok, level, contact, part):
    X, T, p, _ = workload(L, level, contact=L.CONTACT_SMOOTH if contact == "smooth" else L.CONTACT_LINEAR)
    u = squashed_state(X).reshape(-1, 3)
    u[np.abs(X[:, 0]) > part] = 0.0  # only a band is squashed: nodes with few entries at its rim
    u = u.reshape(-1)
    z = np.zeros_like(u)
    f = []
    for _ in range(2):
        g = L.Shell(X, T, p)
        g.set_state(u, z, z)
        f.append(g.eval_forces(u, z, 0.0)[0])
        pairs = np.asarray(g.contact_state()["pairs"]).reshape(-1, 2)
        g.close()
    per_node = np.bincount(T[pairs].reshape(-1), minlength=len(X))
    SEEN.update(int(np.ceil(np.log2(max(32, k)))) for k in per_node if 2 <= k <= 1024)
    assert np.array_equal(f[0].view(np.uint64), f[1].view(np.uint64))


def test_every_network_was_used():
    if not SEEN:
        pytest.skip("runs after the states above")
    assert SEEN == {5, 6, 7, 8, 9, 10}
