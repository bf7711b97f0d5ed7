"""A linked-cell pass over a state with a face that is NaN on one axis.

The face's box is empty there and covers no cell.  On a shell pressed flat in z
the faces' sizes, hence the cells and the distance limit, come from x and y: with
the three nodes of one face NaN in z, the pairs between faces without those nodes
are the ones found without the NaN.  Both walks of the cells (a warp per face for
small shells, a thread and eight lanes above) and a batch's grids."""
import numpy as np
import pytest

from shell_gb300 import lib as L
from shell_gb300.workloads import squashed_state
from tests.common import cell_size_mult_for, physics_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level,copies", [(3, 1), (5, 1), (3, 2)])
def test_pairs_of_the_other_faces(cuda_ok, level, copies):
    X1, T1 = L.icosphere(level)
    p = physics_params(cell_size_mult=cell_size_mult_for(X1, T1, 0.01))
    T = np.concatenate([T1.astype(np.int64) + k * len(X1) for k in range(copies)])
    u = np.concatenate([squashed_state(X1, seed=k) for k in range(copies)])
    z = np.zeros_like(u)

    def context():
        return L.Shell(X1, T1, p) if copies == 1 else L.Batch([(X1, T1)] * copies, [p] * copies)

    def pairs(g, u):
        g.set_state(u, z, z)
        assert g.rebuild_contacts() == 0
        return np.asarray(g.contact_state()["pairs"], dtype=np.int64).reshape(-1, 2)

    g = context()
    clean = pairs(g, u)
    g.close()
    face = int(clean[len(clean) // 3, 0])  # one that has contacts
    bad = u.copy()
    bad[3 * T[face] + 2] = np.nan
    untouched = ~np.isin(T, T[face]).any(axis=1)
    want = clean[untouched[clean].all(axis=1)]
    assert len(clean) > len(want) > 0.9 * len(clean)
    g = context()
    got = pairs(g, bad)
    assert np.array_equal(got[untouched[got].all(axis=1)], want)
    assert not (got == face).any()
    assert np.array_equal(pairs(g, u), clean)  # the context goes on
    g.close()
