"""Launches whose blocks take more than one share of the work, and blocks sized
by the mesh.

A batch of nine level-5 shells has more nodes than one round of the gather's and
of the contact sort's grids (48,640 and 77,824), more cells than one round of the
scan's (2.5 million) and face counts that leave a partly filled warp: it must
equal a shell run alone, which needs one round, bit for bit.  The cavity's node
blocks are 32, 64, 128 or 256 threads: forces within the 1e-12 of the other
cavity tests, on one, two, four and eight spheres in one mesh."""
import numpy as np
import pytest

import oracle as O
from shell_gb300 import lib as L
from tests.common import cell_size_mult_for, physics_params

pytestmark = pytest.mark.gpu


def _bits(x):
    return np.ascontiguousarray(x).view(np.uint64)


def _pinched(X, seed, s=0.0042):
    """The band |x| < 0.3 pressed to a double layer, the rest left round."""
    rng = np.random.default_rng(seed)
    t = np.clip((np.abs(X[:, 0]) - 0.3) / 0.4, 0.0, 1.0)
    u = np.zeros_like(X)
    u[:, 2] = (s - 1.0) * (1.0 - t * t * (3.0 - 2.0 * t)) * X[:, 2]
    return (u + 2e-5 * rng.standard_normal(X.shape)).reshape(-1)


@pytest.mark.parametrize("precision", [L.PREC_FP64, L.PREC_FP32])
def test_batch_beyond_one_round_equals_single_shell(cuda_ok, precision):
    X, T = L.icosphere(5)
    n_shells, h, n = 9, 0.01, 2
    p = physics_params(thickness=h, cell_size_mult=cell_size_mult_for(X, T, h), precision=precision)
    u0s = [_pinched(X, k) for k in range(n_shells)]
    b = L.Batch([(X, T)] * n_shells, [p] * n_shells)
    assert b.V > 77824
    z = np.zeros(3 * b.V)
    b.set_state(np.concatenate(u0s), z, z)
    b.rebuild_contacts()
    rb, _ = b.step(n, np.zeros(n))
    assert rb.steps_done == n
    states = [b.split(x) for x in b.get_state()]
    cb = b.contact_state()
    pairs_b = b.split_pairs(cb["pairs"])
    of = np.searchsorted(b.face_off, cb["pairs"].reshape(-1, 2)[:, 0], side="right") - 1
    b.close()
    for k in (0, n_shells - 1):
        g = L.Shell(X, T, p)
        zz = np.zeros_like(u0s[k])
        g.set_state(u0s[k], zz, zz)
        g.rebuild_contacts()
        g.step(n, np.zeros(n))
        for x, y in zip(g.get_state(), states):
            assert np.array_equal(_bits(x), _bits(y[k]))
        c = g.contact_state()
        assert len(c["pairs"]) > 1000
        assert np.array_equal(np.asarray(c["pairs"]).reshape(-1, 2), pairs_b[k])
        assert np.array_equal(_bits(c["d2"]), _bits(cb["d2"][of == k]))
        g.close()


@pytest.mark.parametrize("copies", [1, 2, 4, 8])
def test_cavity_block_sizes(cuda_ok, copies):
    X1, T1 = L.icosphere(4)
    X = np.concatenate([X1] * copies)
    T = np.concatenate([T1 + k * len(X1) for k in range(copies)]).astype(T1.dtype)
    p = physics_params(contact=False, shell_cavity_contact=1, cavity=L.CAVITY_ELLIPSOID, Rx=1.004, Ry=0.98, Rz=1.001,
                       mu_s_cavity=0.4, mu_d_cavity=0.3, cavity_damping=0.01, cavity_friction_damping=0.01)
    rng = np.random.default_rng(copies)
    u = 2e-3 * rng.standard_normal(X.size)
    v = 0.05 * rng.standard_normal(X.size)
    g, o = L.Shell(X, T, p), O.Oracle(X, T, p, threads=4)
    for s in (g, o):
        s.set_state(u, v, np.zeros_like(u))
    fg = g.eval_forces(u, v, -1e-4)[0]
    fo = o.eval_forces(u, v, -1e-4)[0]
    assert np.linalg.norm(fg - fo) / np.linalg.norm(fo) < 1e-12
    co = o.cavity()["origins"]
    assert np.linalg.norm(g.cavity_origins() - co) / np.linalg.norm(co) < 1e-12
