"""Steps in a cavity at each of the node kernel's block sizes.

One, two, four and eight spheres in one mesh give blocks of 32, 64, 128 and 256
threads.  A step reduces over them: contacts, energies, forces, the largest
move, the kinetic energy; its last block ends the step and starts the next.
Seventeen graph steps (a whole graph and one step of its own) equal direct
launches bit for bit, and the oracle within the bounds of the other cavity
tests (1e-10 for the state, 1e-9 for the sums)."""
import numpy as np
import pytest

import oracle as O
from shell_gb300 import lib as L
from tests.common import physics_params

pytestmark = pytest.mark.gpu

SUMS = ("sum_dt", "sum_area", "sum_volume", "sum_Ekin", "sum_Etens", "sum_Ebend", "sum_Efric", "sum_pcav", "sum_Nc_cav",
        "sum_Ecav")


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("copies", [1, 2, 4, 8])
def test_steps(cuda_ok, copies):
    X1, T1 = L.icosphere(4)
    X = np.concatenate([X1] * copies)
    T = np.concatenate([T1 + k * len(X1) for k in range(copies)]).astype(T1.dtype)
    p = physics_params(contact=False, shell_cavity_contact=1, cavity=L.CAVITY_ELLIPSOID, Rx=1.004, Ry=0.98, Rz=1.001,
                       mu_s_cavity=0.4, mu_d_cavity=0.3, cavity_damping=0.01, cavity_friction_damping=0.01, dt=1e-3)
    rng = np.random.default_rng(copies)
    u = 2e-3 * rng.standard_normal(X.size)
    v = 0.05 * rng.standard_normal(X.size)
    n = 17
    table = -1e-4 * np.linspace(1.0, 2.0, n)
    out = {}
    for name, s in (("graph", L.Shell(X, T, p)), ("direct", L.Shell(X, T, p)), ("oracle", O.Oracle(X, T, p, threads=4))):
        s.set_state(u, v, np.zeros_like(u))
        r, st = s.step(n, table) if name != "direct" else s.step(n, table, use_graph=False)
        assert r.steps_done == n
        out[name] = (r, st, s.get_state(), s.cavity()["origins"] if name == "oracle" else s.cavity_origins())
    (rg, sg, xg, og), (rd, sd, xd, od), (ro, so, xo, oo) = out["graph"], out["direct"], out["oracle"]
    assert sg == sd == so
    assert rg.last.as_dict() == rd.last.as_dict()
    assert all(getattr(rg, k) == getattr(rd, k) for k in SUMS)
    for x, y in zip(xg + (og,), xd + (od,)):
        assert np.array_equal(np.ascontiguousarray(x).view(np.uint64), np.ascontiguousarray(y).view(np.uint64))
    assert rg.last.Nc_cav == ro.last.Nc_cav > 100 * copies
    for k in ("Ekin", "Ecav", "cavity_force", "Efric"):
        assert abs(getattr(rg.last, k) - getattr(ro.last, k)) <= 1e-9 * abs(getattr(ro.last, k)), k
    for k in SUMS:
        assert abs(getattr(rg, k) - getattr(ro, k)) <= 1e-9 * abs(getattr(ro, k)), k
    assert _rel(xg[0], xo[0]) < 1e-10
    assert _rel(og, oo) < 1e-9
