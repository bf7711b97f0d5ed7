"""SMOOTH searches of a batch whose irregular patches' levels are stored in part.

The stored subdivision levels are shared out over the batch's irregular faces: 17
per face for two spheres, 8 for four and more, the last level always among them.
A search goes between the stored levels and those beyond as its point moves.  Each shell's pairs,
squared distances, search coordinates and state are those of the shell alone (all
34 levels stored) bit for bit, after a list build and after steps."""
import numpy as np
import pytest

from shell_gb300 import lib as L
from shell_gb300.workloads import squashed_state
from tests.common import cell_size_mult_for, physics_params

pytestmark = pytest.mark.gpu


def _bits(x):
    return np.ascontiguousarray(x).view(np.uint64)


def _snapshot(g):
    c = g.contact_state()
    return list(g.get_state()), np.asarray(c["pairs"], dtype=np.int64).reshape(-1, 2), c["d2"], g.contact_coords()


@pytest.mark.parametrize("copies", [2, 4, 40])
def test_batch_equals_single(cuda_ok, copies):
    X, T = L.icosphere(2)
    p = physics_params(shell_shell_contact=L.CONTACT_SMOOTH, cell_size_mult=cell_size_mult_for(X, T, 0.01))
    us = [squashed_state(X, seed=k) for k in range(copies)]
    b = L.Batch([(X, T)] * copies, [p] * copies)
    z = np.zeros(3 * b.V)
    b.set_state(np.concatenate(us), z, z)
    b.rebuild_contacts()
    first = _snapshot(b)
    b.step(3, np.zeros(3))
    last = _snapshot(b)
    for k in (0, copies - 1):
        g = L.Shell(X, T, p)
        zz = np.zeros_like(us[k])
        g.set_state(us[k], zz, zz)
        g.rebuild_contacts()
        for snap in (first, last):
            (state, pairs, d2, x), (sg, pg, dg, xg) = snap, _snapshot(g)
            mine = (pairs[:, 0] >= b.face_off[k]) & (pairs[:, 0] < b.face_off[k + 1])
            assert len(pg) > 500
            assert np.array_equal(pairs[mine] - b.face_off[k], pg)
            assert np.array_equal(_bits(d2[mine]), _bits(dg))
            assert np.array_equal(_bits(x[mine]), _bits(xg))
            for q, s in zip(state, sg):
                assert np.array_equal(_bits(b.split(q)[k]), _bits(s))
            g.step(3, np.zeros(3))
        g.close()
    b.close()
