"""SMOOTH contact on meshes with many irregular vertices, against the oracle.

The power forms of irregular patches are kept for as many subdivision levels as
the number of irregular faces allows: all 34 on a sphere, a few on a mesh with
hundreds of irregular faces, none with thousands; deeper points are subdivided
in the search.  The pair list, the squared distances and the searches'
coordinates must be the oracle's bit for bit in each case."""
import numpy as np
import pytest

from shell_gb300 import lib as L
import oracle as O
from tests.common import cell_size_mult_for, midpoint_refine, physics_params

pytestmark = pytest.mark.gpu


def flipped(level, flips, seed):
    """An icosphere with random edges flipped (valences 4 to 9), refined once."""
    X, T = L.icosphere(level)
    T = np.array(T, dtype=np.int64)
    rng = np.random.default_rng(seed)
    val = np.bincount(T.ravel())
    faces_of = {(int(t[k]), int(t[(k + 1) % 3])): f for f, t in enumerate(T) for k in range(3)}
    done = 0
    while done < flips:
        f, k = int(rng.integers(len(T))), int(rng.integers(3))
        p, q, r = int(T[f][k]), int(T[f][(k + 1) % 3]), int(T[f][(k + 2) % 3])
        g = faces_of[(q, p)]
        s = [int(x) for x in T[g] if x not in (p, q)][0]
        if val[p] <= 4 or val[q] <= 4 or val[r] >= 9 or val[s] >= 9 or (r, s) in faces_of or (s, r) in faces_of:
            continue
        for t in (T[f], T[g]):
            for m in range(3):
                del faces_of[(int(t[m]), int(t[(m + 1) % 3]))]
        T[f], T[g] = (r, s, q), (s, r, p)
        for h in (f, g):
            for m in range(3):
                faces_of[(int(T[h][m]), int(T[h][(m + 1) % 3]))] = h
        val[p] -= 1
        val[q] -= 1
        val[r] += 1
        val[s] += 1
        done += 1
    X, T = midpoint_refine(X, T)
    return np.ascontiguousarray(X, dtype=np.float64), np.ascontiguousarray(T, dtype=np.uint32)


@pytest.mark.parametrize("level,flips,levels", [(2, 20, (1, 33)), (3, 400, (0, 0))])
def test_pairs_and_coordinates(cuda_ok, level, flips, levels):
    X, T = flipped(level, flips, seed=level)
    irregular = int(np.sum(np.any(np.bincount(T.ravel())[T] != 6, axis=1)))
    assert levels[0] <= min(34, 2048 // irregular) <= levels[1]
    rng = np.random.default_rng(31)
    u = np.zeros_like(X)
    u[:, 2] = (0.0042 - 1.0) * X[:, 2]
    u = (u + 2e-5 * rng.standard_normal(X.shape)).reshape(-1)
    v = 0.02 * rng.standard_normal(u.shape)
    p = physics_params(shell_shell_contact=L.CONTACT_SMOOTH, cell_size_mult=cell_size_mult_for(X, T, 0.01))
    g, o = L.Shell(X, T, p), O.Oracle(X, T, p, threads=8)
    for s in (g, o):
        s.set_state(u, v, np.zeros_like(u))
        s.eval_forces(u, v, 0.0)
    cg, co = g.contact_state(), o.contact_state()
    assert len(co["pairs"]) > 500
    assert np.array_equal(cg["pairs"], co["pairs"])
    assert np.array_equal(cg["d2"].view(np.uint64), co["d2"].view(np.uint64))
    assert np.array_equal(g.contact_coords().view(np.uint64), o.contact_coords().view(np.uint64))
    g.close()
