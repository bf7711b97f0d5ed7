"""Per-face and per-node fields after a graph run that ends before its last step.

Steps of a graph alternate between two sets of the per-face measurements.  A run
may stop after any of them: by a stopping criterion, by a problem.  The fields
read afterwards must be those of the step that ended the run, the totals and sums
those of the steps made: all as with direct launches, bit for bit."""
import numpy as np
import pytest

from shell_gb300 import lib as L
from tests.common import cell_size_mult_for, physics_params

pytestmark = pytest.mark.gpu

N, DT = 20, 1e-3


def _bits(x):
    return np.ascontiguousarray(x).view(np.uint64)


def _pressed(X, seed):
    rng = np.random.default_rng(seed)
    u = np.zeros_like(X)
    u[:, 2] = (0.0042 - 1.0) * X[:, 2]
    return (u + 2e-5 * rng.standard_normal(X.shape)).reshape(-1)


def _run(kind, last, use_graph, graph_first):
    """A run of N steps that ends after `last` of them, and what a caller can read then."""
    X, T = L.icosphere(2)
    rng = np.random.default_rng(7)
    kw = dict(dt=DT, thickness=0.02)
    table = -1e-4 * (1.0 + 0.1 * np.arange(N))
    v0 = 0.05 * rng.standard_normal(X.size)
    u0 = 1e-3 * rng.standard_normal(X.size)
    if kind == "contact":
        u0 = _pressed(X, 3)
        kw.update(cell_size_mult=cell_size_mult_for(X, T, 0.02), dt=1e-4)
    elif kind == "cavity":
        kw.update(contact=False, shell_cavity_contact=1, cavity=L.CAVITY_ELLIPSOID, Rx=1.004, Ry=0.98, Rz=1.001,
                  mu_s_cavity=0.4, mu_d_cavity=0.3)
    elif kind == "problem":
        # step `last` is driven hard enough to move beyond half the thickness
        kw.update(cell_size_mult=cell_size_mult_for(X, T, 0.02), stop_on_problem=1, dt=1e-2)
        v0 *= 0.1
        table[last - 1] = -20.0
    else:
        kw.update(contact=False, precision=L.PREC_FP32 if kind == "fp32" else L.PREC_FP64)
    p = physics_params(**kw)
    if kind == "batch":
        g = L.Batch([(X, T)] * 3, [p] * 3, [1.0, 0.5, 2.0])
        u0, v0 = np.tile(u0, 3), np.tile(v0, 3)
    else:
        g = L.Shell(X, T, p)
    g.set_state(u0, v0, np.zeros_like(u0))
    if kind in ("contact", "problem"):
        g.rebuild_contacts()
    if graph_first:  # a whole graph before the one that stops
        g.step(16, np.full(16, -1e-4), use_graph=use_graph)
    if kind != "problem":
        g.set_stop_function("t > %r" % (g.get_time()[0] + (last - 0.5) * kw["dt"]))
    r, st = g.step(N, table, use_graph=use_graph)
    out = {"report": [getattr(r, k) for k in ("steps_done", "worst_problem", "stopped", "time", "sum_dt", "sum_area",
                                              "sum_volume", "sum_Nc", "sum_Ekin", "sum_Etens", "sum_Ebend", "sum_Eself",
                                              "sum_Efric", "sum_kGauss", "sum_kMean", "sum_pcav", "sum_Nc_cav",
                                              "sum_Ecav")] + sorted(r.last.as_dict().items()),
           "status": st}
    for k, x in zip("uva", g.get_state()):
        out[k] = _bits(x)
    for k, x in list(g.element_fields().items()) + list(g.node_fields().items()):
        out["field " + k] = _bits(x)
    g.close()
    return out


@pytest.mark.parametrize("kind", ["plain", "fp32", "contact", "cavity", "batch", "problem"])
@pytest.mark.parametrize("last", range(1, 18))
def test_fields_of_the_last_step(cuda_ok, kind, last):
    d = _run(kind, last, use_graph=False, graph_first=last == 3)
    g = _run(kind, last, use_graph=True, graph_first=last == 3)
    assert d["report"][0] == last
    assert d["report"][1] == 2 if kind == "problem" else d["report"][2] == 1  # 2: LARGE_DISP
    for k in d:
        if k in ("report", "status"):
            assert d[k] == g[k], k
        else:
            assert np.array_equal(d[k], g[k]), k


def test_list_after_a_problem(cuda_ok):
    """The step that a problem ends may have made a linked-cell pass due: graph runs make it
    when they report or the list is read, as direct launches make it at the end of the step."""
    X, T = L.icosphere(3)
    p = physics_params(cell_size_mult=cell_size_mult_for(X, T, 0.01), stop_on_problem=1)
    u0 = _pressed(X, 3)
    # the middle band set in motion: half the thickness in one step
    v0 = np.zeros_like(X)
    v0[np.abs(X[:, 0]) < 0.3, 2] = 60.0
    out = []
    for use_graph, read in ((False, False), (True, False), (True, True)):
        g = L.Shell(X, T, p)
        g.set_state(u0, v0.reshape(-1), np.zeros_like(u0))
        g.rebuild_contacts()
        if read:  # the list is read before the steps are collected
            g.step_collect()  # the report starts here, as step() lets it
            g.upload_pressure_table(np.zeros(N))
            g.step_enqueue(N)
            g.contact_state()
            r, st = g.step_collect()
        else:
            r, st = g.step(N, np.zeros(N), use_graph=use_graph)
        assert r.worst_problem == 2 and r.steps_done < N  # LARGE_DISP
        c = g.contact_state()
        one = [r.steps_done, r.n_rebuilds, r.du_sum, c["du_sum"], c["pairs"], c["stick"], _bits(c["origin"]), _bits(c["d2"])]
        r, _ = g.step(2, np.zeros(2), use_graph=use_graph)
        one += [r.steps_done, r.n_rebuilds] + [_bits(x) for x in g.get_state()]
        out.append(one)
        g.close()
    assert out[0][1] >= 2  # the build, the predictor's pass, the corrector's
    for k, (a, b, c) in enumerate(zip(*out)):
        assert np.array_equal(a, b) and np.array_equal(a, c), k
