"""Timed workloads of the framework: what a user has it do through shell_gb300.lib.

Every workload is a shell (or a batch of shells) of the benchmark family: a unit
sphere triangulated at frequency n (20 n^2 faces: n = 8, 16, 32, 64, 128 are the
icosphere levels 3 to 7; other n give ragged sizes), orthotropic material, h/R
about 0.01, seeded imperfections, an external pressure ramp.  A program that owns
the state on the host (page-locked buffers) sets it, advances it and reads it
back, as a driver of the C ABI does; the number of steps in between is what
differs between an interactive step and a long run.

The oracle part (`exact`) restates the explicit step in float64 torch from the
mechanics: Loop basis at the face centroid, Koiter strains from displacement
derivatives, lumped masses, Newmark, cavity and self-contact penalty forces with
slip-stick friction.  It uses nothing of the package.
"""
import math

import numpy as np
import torch

from shell_gb300 import lib as L

H = 0.01          # thickness of the single shells
DT = 1e-4
ALPHA = 0.05      # mass-proportional damping
RAMP_STEPS = 20000
MU = 0.3
STEP_FLOPS = 1400.0   # floating-point operations of one face's forces in one step
PAIR_FLOPS = 1000.0   # closest points of one contact pair: 9 edge-edge, 6 vertex-face
SEARCH_FLOPS = 4 * 1100.0  # limit-surface search of a pair: a few evaluations of two quartic patches


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # one step of a small shell driven from the host: the smallest call
        {"name": "step_small", "kind": "step", "n": 8, "steps": 1, "prec": "fp64", "contact": "linear"},
        # the reference's own level-3 run, a stretch between two outputs
        {"name": "run_small", "kind": "step", "n": 8, "steps": 256, "prec": "fp64", "contact": "linear"},
        # forces and accelerations at a given state, ragged mesh (host program integrates itself)
        {"name": "forces_ragged", "kind": "forces", "n": 37, "prec": "fp64", "contact": "linear"},
        # a shell growing into an ellipsoidal cavity with wall friction, ragged mesh
        {"name": "cavity_ragged", "kind": "cavity", "n": 21, "steps": 100, "prec": "fp64"},
        # the benchmark's shell, one step with host state in and out
        {"name": "step_level6", "kind": "step", "n": 64, "steps": 1, "prec": "fp64", "contact": "linear"},
        # the same, a stretch of a long run
        {"name": "run_level6", "kind": "step", "n": 64, "steps": 64, "prec": "fp64", "contact": "linear"},
        # the largest single shell, FP32 forces
        {"name": "run_level7_fp32", "kind": "step", "n": 128, "steps": 32, "prec": "fp32", "contact": "none"},
        # parameter study: 256 shells of mixed sizes and materials, FP32 forces, own self-contact each
        {"name": "ensemble_fp32", "kind": "ensemble", "shells": 256, "steps": 16},
        # dynamic relaxation of a batch with a residual check (the warm-start study), FP64
        {"name": "relax_batch", "kind": "relax", "n": 16, "shells": 32, "steps": 100},
        # a shell folded onto itself everywhere: list build and contact-heavy steps
        {"name": "folded_linear", "kind": "folded", "n": 64, "steps": 8, "contact": "linear"},
        # the same with limit-surface contact
        {"name": "folded_smooth", "kind": "folded", "n": 32, "steps": 4, "contact": "smooth"},
        # gradients of the warm-start network of the level-4 study
        {"name": "network_gradients", "kind": "network", "rows": 256, "hidden": 512, "outputs": 7686},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "forces", "cavity", "ensemble", "relax", "folded", "folded_smooth",
                       "network"])
    if kind == "step":
        prec = rng.choice(["fp64", "fp64", "fp32"])
        n = _log_int(rng, 8, 100)
        return {"kind": "step", "n": n, "steps": rng.choice([1, 7, 16, 50, _log_int(rng, 8, 128)]), "prec": prec,
                "contact": rng.choice(["linear", "linear", "none"])}
    if kind == "forces":
        return {"kind": "forces", "n": _log_int(rng, 8, 100), "prec": rng.choice(["fp64", "fp32"]),
                "contact": rng.choice(["linear", "none"])}
    if kind == "cavity":
        return {"kind": "cavity", "n": _log_int(rng, 8, 48), "steps": _log_int(rng, 20, 100), "prec": "fp64"}
    if kind == "ensemble":
        return {"kind": "ensemble", "shells": _log_int(rng, 16, 192), "steps": rng.choice([8, 16, 21])}
    if kind == "relax":
        return {"kind": "relax", "n": _log_int(rng, 8, 20), "shells": _log_int(rng, 8, 32),
                "steps": _log_int(rng, 50, 100)}
    if kind == "folded":
        return {"kind": "folded", "n": _log_int(rng, 12, 60), "steps": rng.randint(2, 8), "contact": "linear"}
    if kind == "folded_smooth":
        return {"kind": "folded", "n": _log_int(rng, 10, 30), "steps": rng.randint(1, 4), "contact": "smooth"}
    return {"kind": "network", "rows": rng.randint(17, 256), "hidden": rng.choice([64, 128, 256, 512]),
            "outputs": 3 * _log_int(rng, 642, 2562)}


# ----------------------------------------------------------------- inputs --
_MESHES = {}


def _sphere(n):
    """Unit sphere, 20 n^2 faces, 10 n^2 + 2 nodes, outward oriented, turned so that no face is level."""
    if n in _MESHES:
        return _MESHES[n]
    g = (1 + math.sqrt(5)) / 2
    P = np.array([(0, s1, s2 * g) for s1 in (-1, 1) for s2 in (-1, 1)], float)
    P = np.concatenate([P, P[:, [1, 2, 0]], P[:, [2, 0, 1]]]) / math.sqrt(1 + g * g)
    edge = min(np.linalg.norm(P[0] - P[k]) for k in range(1, 12)) * 1.01
    tri = [(a, b, c) for a in range(12) for b in range(a + 1, 12) for c in range(b + 1, 12)
           if max(np.linalg.norm(P[a] - P[b]), np.linalg.norm(P[b] - P[c]), np.linalg.norm(P[a] - P[c])) < edge]
    i, j = np.meshgrid(np.arange(n + 1), np.arange(n + 1), indexing="ij")
    keep = i + j <= n
    idx = -np.ones((n + 1, n + 1), np.int64)
    idx[keep] = np.arange(keep.sum())
    bi, bj = i[keep], j[keep]
    up = (bi + bj < n)
    dn = (bi + bj < n - 1)
    F1 = np.stack([idx[bi[up], bj[up]], idx[bi[up] + 1, bj[up]], idx[bi[up], bj[up] + 1]], 1)
    F2 = np.stack([idx[bi[dn] + 1, bj[dn]], idx[bi[dn] + 1, bj[dn] + 1], idx[bi[dn], bj[dn] + 1]], 1)
    nodes, faces, off = [], [], 0
    for a, b, c in tri:
        if np.dot(np.cross(P[b] - P[a], P[c] - P[a]), P[a]) < 0:
            b, c = c, b
        X = ((n - bi - bj)[:, None] * P[a] + bi[:, None] * P[b] + bj[:, None] * P[c]) / n
        nodes.append(X / np.linalg.norm(X, axis=1, keepdims=True))
        faces.append(np.concatenate([F1, F2]) + off)
        off += len(X)
    X, F = np.concatenate(nodes), np.concatenate(faces)
    _, first, inv = np.unique(np.round(X * 1e7).astype(np.int64), axis=0, return_index=True, return_inverse=True)
    rot = np.linalg.qr(np.random.default_rng(7).standard_normal((3, 3)))[0]
    rot *= np.linalg.det(rot)
    out = np.ascontiguousarray(X[first] @ rot.T), np.ascontiguousarray(inv.reshape(-1)[F].astype(np.uint32))
    _MESHES[n] = out
    return out


def _extent(X, T):
    P = X[T]
    return float((P.max(axis=1) - P.min(axis=1)).max(axis=1).mean())


def _p_cl(e1, e2, nu12, h):
    nu = math.sqrt(nu12 * nu12 * e2 / e1)
    return 2 * math.sqrt(e1 * e2) * h * h / math.sqrt(3 * (1 - nu * nu))


def _material(e1=1.0, e2=0.5, nu=0.3, g=0.35, h=H, alpha=ALPHA, dt=DT):
    return {"e1": e1, "e2": e2, "nu": nu, "g": g, "h": h, "alpha": alpha, "dt": dt}


def _modes(X, rng, amp):
    """A smooth random vector field of low order."""
    A, B = rng.standard_normal((3, 3)), rng.standard_normal((3, 3))
    return amp * (X @ A.T + (X * X[:, [1, 2, 0]]) @ B.T)


def _inputs(case, seed):
    """Everything a pass starts from, from the seed alone (numpy)."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    d = {}
    if kind == "network":
        dims = [8] + [case["hidden"]] * 4 + [case["outputs"]]
        d["dims"] = dims
        d["params"] = [((rng.standard_normal((o, i)) * math.sqrt(2.0 / i)).astype(np.float32),
                        (0.05 * rng.standard_normal(o)).astype(np.float32)) for i, o in zip(dims[:-1], dims[1:])]
        d["X"] = rng.standard_normal((case["rows"], 8)).astype(np.float32)
        d["T"] = rng.standard_normal((case["rows"], case["outputs"])).astype(np.float32)
        return d
    if kind == "ensemble":
        mats, meshes, scale, u = [], [], [], []
        for n in np.random.default_rng(case["shells"]).integers(8, 33, case["shells"]):  # sizes belong to the case
            X, T = _sphere(int(n))
            r, h = math.exp(rng.uniform(math.log(0.2), math.log(5.0))), math.exp(rng.uniform(math.log(0.005), math.log(0.05)))
            amp, s = math.exp(rng.uniform(math.log(1e-4), math.log(3e-3))), rng.uniform(1.2, 3.0)
            e1, e2 = math.sqrt(r), 1 / math.sqrt(r)
            mats.append(_material(e1, e2, 0.3, 0.35, h))
            meshes.append((X, T))
            scale.append(s * _p_cl(e1, e2, 0.3, h))
            u.append(amp * rng.standard_normal((len(X), 1)) * X)
        steps = case["steps"]
        k0 = int(rng.integers(0, RAMP_STEPS - steps))
        table = -np.arange(k0 + 1, k0 + steps + 1) / RAMP_STEPS
    elif kind == "relax":
        X, T = _sphere(case["n"])
        mats, meshes, scale, u = [], [], [], []
        for _ in range(case["shells"]):
            r, nu, g = math.exp(rng.uniform(math.log(0.2), math.log(5.0))), rng.uniform(0.25, 0.35), rng.uniform(0.3, 0.45)
            h, s, c = math.exp(rng.uniform(math.log(0.005), math.log(0.05))), rng.uniform(0.15, 0.5), rng.standard_normal(3)
            e1, e2 = math.sqrt(r), 1 / math.sqrt(r)
            x, y, z = X.T
            w = 0.3 * h * (c[0] * (3 * z * z - 1) / 2 + c[1] * math.sqrt(3) * x * z + c[2] * x * (5 * z * z - 1) / 2)
            mats.append(_material(e1, e2, nu, g, h, alpha=1.0, dt=64e-3 / case["n"]))
            meshes.append((X * (1 + w[:, None]), T))
            scale.append(s * _p_cl(e1, e2, nu, h))
            u.append(1e-3 * h * rng.standard_normal((len(X), 1)) * X)
        table = np.full(case["steps"], -1.0)
    else:
        X, T = _sphere(case["n"])
        mats, meshes, scale = [_material()], [(X, T)], [1.0]
        steps = case.get("steps", 1)
        if kind == "folded":
            # flattened to a double layer (gap about 2 s |z|); the layers slide past each other
            w = (0.0042 - 1.0) * X[:, 2:3] * np.array([[0.0, 0.0, 1.0]])
            u = [w + 2e-5 * rng.standard_normal(X.shape)]
            table = np.zeros(steps)
        else:
            u = [1e-3 * rng.standard_normal((len(X), 1)) * X]
            k0 = int(rng.integers(0, RAMP_STEPS // 2))
            table = -2 * _p_cl(1.0, 0.5, 0.3, H) * np.arange(k0 + 1, k0 + steps + 1) / RAMP_STEPS
    V = [len(X) for X, _ in meshes]
    v = [np.zeros((k, 3)) if kind == "relax" else _modes(X, rng, 1e-3) for k, (X, _) in zip(V, meshes)]
    if kind == "folded":
        X = meshes[0][0]
        v = [np.sign(X[:, 2:3]) * np.array([[0.03, 0.01, 0.0]]) + 2e-3 * rng.standard_normal(X.shape)]
    if kind == "cavity":
        v = [0.05 * rng.standard_normal(meshes[0][0].shape)]
    d.update(mats=mats, meshes=meshes, scale=np.array(scale), table=np.asarray(table, float),
             u=np.concatenate(u).reshape(-1), v=np.concatenate(v).reshape(-1))
    return d


# the ellipsoidal cavity of the cavity case: in touch with the imperfect sphere
_CAVITY = {"R": (1.004, 0.998, 1.001), "mu_s": 0.4, "mu_d": 0.3, "damping": 0.01, "fric_damping": 0.01}


def _params(m, X, T, contact, prec, **kw):
    return L.default_params(shell_mass_density=1.0, shell_young_modulus=m["e1"], shell_young_modulus2=m["e2"],
                            shell_poisson_ratio=m["nu"], shell_shear_modulus=m["g"], thickness=m["h"],
                            damping_alpha=m["alpha"], dt=m["dt"], shell_shell_contact=contact, mu_s=MU, mu_d=MU,
                            cell_size_mult=2 * m["h"] / _extent(X, T), precision=prec, **kw)


def _pinned(n):
    return torch.zeros(n, dtype=torch.float64).pin_memory()


# ---------------------------------------------------------------- prepare --
def prepare(case, seed):
    d = _inputs(case, seed)
    if case["kind"] == "network":
        net = L.MLP(d["dims"], max_batch=256, seed=1)
        net.set_params(d["params"])
        return {"case": case, "net": net, "X": d["X"], "T": d["T"]}
    kind = case["kind"]
    prec = L.PREC_FP32 if case.get("prec") == "fp32" or kind == "ensemble" else L.PREC_FP64
    mode = {"linear": L.CONTACT_LINEAR, "smooth": L.CONTACT_SMOOTH, "none": L.CONTACT_NONE}[
        case.get("contact", "linear" if kind == "ensemble" else "none")]
    kw = {}
    if kind == "cavity":
        c = _CAVITY
        kw = dict(shell_cavity_contact=1, cavity=L.CAVITY_ELLIPSOID, Rx=c["R"][0], Ry=c["R"][1], Rz=c["R"][2],
                  mu_s_cavity=c["mu_s"], mu_d_cavity=c["mu_d"], cavity_damping=c["damping"],
                  cavity_friction_damping=c["fric_damping"])
    params = [_params(m, X, T, mode, prec, **kw) for m, (X, T) in zip(d["mats"], d["meshes"])]
    if kind in ("ensemble", "relax"):
        sh = L.Batch(d["meshes"], params, pressure_scale=d["scale"])
    else:
        sh = L.Shell(*d["meshes"][0], params[0])
    hold = [_pinned(3 * sh.V) for _ in range(6)]
    buf = [t.numpy() for t in hold]
    buf[0][:], buf[1][:], buf[2][:] = d["u"], d["v"], 0.0
    sh.apply_initial_conditions(buf[0], 0.0, float(d["table"][0]))  # first candidate list, volume
    return {"case": case, "sh": sh, "hold": hold, "in": buf[:3], "out": buf[3:], "table": d["table"]}


# -------------------------------------------------------------------- run --
def _report(r):
    e = r.last
    return np.array([e.Etens, e.Ebend, e.Eself, e.Efric, e.Ekin, e.area, e.kGauss, e.kMean, e.Ecav])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "network":
        loss, dW, db = state["net"].gradients(state["X"], state["T"])
        return [np.array([loss])] + dW + db
    sh, (u, v, a) = state["sh"], state["in"]
    if kind == "forces":
        # (the list keeps its own trigger; the displacement's velocity is v)
        f, acc, e, _ = sh.eval_forces(u, v, float(state["table"][0]))
        return [f, acc, np.array([e["Etens"], e["Ebend"], e["area"]])]
    sh.set_state(u, v, a)
    if kind == "folded":
        sh.set_contact_state(np.zeros((0, 2), np.uint32))
        sh.rebuild_contacts()
    if kind == "cavity":
        zero = np.zeros(3 * sh.V)  # no friction springs yet
        sh.lib.shl_set_cavity_origins(sh.h, zero.ctypes.data)
    r, _ = sh.step(len(state["table"]), state["table"])
    out = state["out"]
    sh.get_state(out)
    counts = np.array([r.steps_done, r.last.Nc, r.last.Nc_cav], dtype=np.int64)
    res = [out[0], out[1], out[2], _report(r), counts]
    if kind == "relax":
        res.append(sh.residual(float(state["table"][-1]), L.RESIDUAL_FP64))
    return res


# ------------------------------------------------------------------- work --
def work(case):
    kind = case["kind"]
    if kind == "network":
        dims = [8] + [case["hidden"]] * 4 + [case["outputs"]]
        w = sum(i * o for i, o in zip(dims[:-1], dims[1:]))
        return {"bytes": 4.0 * (2 * w + case["rows"] * (8 + case["outputs"])), "flops": 6.0 * case["rows"] * w}
    steps = case.get("steps", 1)
    # a batch's sphere frequencies are uniform in 8..32
    faces = {"ensemble": case.get("shells", 0) * 20 * 462.0, "relax": case.get("shells", 0) * 20.0 * case.get("n", 0) ** 2}.get(
        kind, 20.0 * case.get("n", 0) ** 2)
    nodes = faces / 2
    word = 4 if case.get("prec") == "fp32" or kind == "ensemble" else 8
    # face constants and patch ids once, the state in and out, masses and reference positions
    nbytes = faces * (37 * word + 12 * 4) + nodes * 8 * (9 + 9 + 9)
    flops = faces * STEP_FLOPS * steps
    if kind == "folded":
        n = case["n"]
        edge, area = 1.11 / n, 2 * math.pi / faces
        reach = 1.04 * H + (edge if case["contact"] == "smooth" else 0.0)
        pairs = 0.5 * faces * math.pi * (reach + 0.9 * edge) ** 2 / area
        per = SEARCH_FLOPS if case["contact"] == "smooth" else PAIR_FLOPS
        nbytes += pairs * 8 * (steps + 1)
        flops += pairs * per * (steps + 1)
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------ exact --
_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(x, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=dtype, device=_DEV)


# The regular patch at its centroid: twelve box splines at lattice offsets
# (p, q) from the face's first node, as (1/12) sum c u^i v^j w^k.
_BOX = {
    (0, -1): "1400 2310", (-1, 0): "1400 2301",
    (1, -1): "1400 2301 6310 6211 c220 6121 6130 2031 1040",
    (0, 0): "6400 o301 o202 8103 1004 o310 s211 t112 6013 o220 t121 c022 8130 6031 1040",
    (-1, 1): "1400 6301 c202 6103 1004 2310 6211 6112 2013",
    (2, -1): "2130 1040",
    (1, 0): "1400 6301 c202 6103 1004 8310 t211 t112 8013 o220 s121 o022 o130 o031 6040",
    (0, 1): "1400 8301 o202 o103 6004 6310 t211 s112 o013 c220 t121 o022 6130 8031 1040",
    (-1, 2): "2103 1004", (2, 0): "2031 1040",
    (1, 1): "2103 1004 6112 6013 6121 c022 2130 6031 1040", (0, 2): "1004 2013",
}
_DIG = {"c": 12, "o": 24, "t": 36, "s": 60}


def _poly(terms, d):
    """Value at u = v = w = 1/3 of the derivative d = (in u, in v, in w) of the polynomial."""
    r = 0.0
    for t in terms.split():
        c, e = float(_DIG.get(t[0], 0) or int(t[0])), [int(x) for x in t[1:]]
        for ex, k in zip(e, d):
            for q in range(k):
                c *= ex - q
            c *= (1.0 / 3.0) ** max(ex - k, 0) if ex >= k else 0.0
        r += c
    return r / 12.0


def _box_basis():
    """Per lattice offset: value, d/dv, d/dw, d2/dv2, d2/dw2, d2/dvdw at the centroid."""
    out = {}
    for p, t in _BOX.items():
        f = lambda a, b, c: _poly(t, (a, b, c))  # noqa: E731
        out[p] = np.array([f(0, 0, 0), f(0, 1, 0) - f(1, 0, 0), f(0, 0, 1) - f(1, 0, 0),
                           f(0, 2, 0) - 2 * f(1, 1, 0) + f(2, 0, 0), f(0, 0, 2) - 2 * f(1, 0, 1) + f(2, 0, 0),
                           f(0, 1, 1) - f(1, 1, 0) - f(1, 0, 1) + f(2, 0, 0)])
    return out


def _patch_basis(N):
    """(N + 6) x 6 basis at the centroid; slots: a, b, c, ring of a after c, d, two around b, two around c."""
    ring = [1, 2] + list(range(3, N + 1))
    d, b0, b1, c0, c1 = N + 1, N + 2, N + 3, N + 4, N + 5
    B = np.zeros((N + 6, 6))
    box = _box_basis()
    if N == 6:
        at = {(0, 0): 0, (1, 0): 1, (0, 1): 2, (-1, 1): 3, (-1, 0): 4, (0, -1): 5, (1, -1): 6, (1, 1): d, (2, 0): b0,
              (2, -1): b1, (0, 2): c0, (-1, 2): c1}
        for p, s in at.items():
            B[s] = box[p]
        return B

    def edge(p, q, o1, o2):
        w = np.zeros(N + 6)
        w[[p, q]], w[[o1, o2]] = 0.375, 0.125
        return w

    def vert(c, rim):
        w = np.zeros(N + 6)
        w[c] = 0.625
        w[rim] = 0.0625
        return w

    beta = (0.625 - (0.375 + 0.25 * math.cos(2 * math.pi / N)) ** 2) / N
    va = np.zeros(N + 6)
    va[0] = 1 - N * beta
    va[ring] = beta
    last, third = ring[N - 1], ring[2]
    # the middle child of one Loop step: corners bc, ca, ab (its v and w axes run against the parent's)
    child = {(0, 0): edge(1, 2, 0, d), (1, 0): edge(2, 0, 1, third), (0, 1): edge(0, 1, 2, last),
             (1, 1): va, (-1, 0): edge(1, d, 2, b0), (0, -1): edge(2, d, 1, c0), (1, -1): vert(2, [0, 1, d, c0, c1, third]),
             (-1, 1): vert(1, [2, 0, last, b1, b0, d]), (2, -1): edge(2, third, 0, c1), (-1, 2): edge(1, last, 0, b1),
             (2, 0): edge(0, third, 2, ring[3 % N]), (0, 2): edge(0, last, 1, ring[N - 2])}
    jac = np.array([1.0, -2, -2, 4, 4, 4])
    for p, w in child.items():
        B += w[:, None] * (jac * box[p])[None, :]
    return B


def _patches(T, V):
    """Per valence of the face's irregular corner (6: none): face ids and patch node ids."""
    T = np.asarray(T, np.int64)
    frm, to, opp = T.reshape(-1), T[:, [1, 2, 0]].reshape(-1), T[:, [2, 0, 1]].reshape(-1)
    key = frm * V + to
    order = np.argsort(key)
    skey, sopp = key[order], opp[order]

    def turn(c, x):
        return sopp[np.searchsorted(skey, c * V + x)]

    val = np.bincount(T.reshape(-1), minlength=V)
    irr = val[T] != 6
    first = np.where(irr.any(1), irr.argmax(1), 0)
    R = np.stack([T[np.arange(len(T)), (first + k) % 3] for k in range(3)], 1)
    out = {}
    for N in np.unique(val[R[:, 0]]):
        ids = np.nonzero(val[R[:, 0]] == N)[0]
        a, b, c = R[ids].T
        ring = [b, c]
        for _ in range(int(N) - 2):
            ring.append(turn(a, ring[-1]))
        b1 = turn(b, ring[-1])
        b0 = turn(b, b1)
        dd = turn(b, b0)
        c0 = turn(c, dd)
        c1 = turn(c, c0)
        out[int(N)] = (ids, np.stack([a, b, c] + ring[2:] + [dd, b0, b1, c0, c1], 1))
    return out


def _dot(a, b):
    return (a * b).sum(-1)


class _Exact:
    """The shells' mechanics in float64: reference constants per face, forces and measurements."""

    def __init__(self, d):
        parts, off, foff, per_mesh = {}, 0, 0, {}
        X, T, fm = [], [], []
        for k, (x, t) in enumerate(d["meshes"]):
            if t.shape not in per_mesh:
                per_mesh[t.shape] = _patches(t, len(x))
            for N, (ids, P) in per_mesh[t.shape].items():
                parts.setdefault(N, []).append((ids + foff, P + off))
            X.append(x)
            T.append(t.astype(np.int64) + off)
            fm.append(np.full(len(t), k))
            off, foff = off + len(x), foff + len(t)
        self.X, self.T, self.V, self.F = _t(np.concatenate(X)), _t(np.concatenate(T), torch.int64), off, foff
        self.node_shell = _t(np.repeat(np.arange(len(X)), [len(x) for x in X]), torch.int64)
        shell = np.concatenate(fm)
        m = {k: np.array([q[k] for q in d["mats"]]) for k in d["mats"][0]}
        self.m, self.dt = m, float(m["dt"][0])
        self.groups = []
        nu21 = m["e2"] * m["nu"] / m["e1"]
        Kall, Dall = m["h"] / (1 - m["nu"] * nu21), m["h"] ** 3 / (12 * (1 - m["nu"] * nu21))
        self.K = Kall
        M, C = torch.zeros(self.V, **_F64), torch.zeros(self.V, **_F64)
        for N, lst in parts.items():
            ids, P = np.concatenate([i for i, _ in lst]), np.concatenate([p for _, p in lst])
            q = {"ids": _t(ids, torch.int64), "P": _t(P, torch.int64), "B": _t(_patch_basis(N))}
            g = lambda k: _t(m[k][shell[ids]])  # noqa: E731
            q["K"], q["D"] = _t(Kall[shell[ids]]), _t(Dall[shell[ids]])
            q["ps"] = _t(d["scale"][shell[ids]])
            G = torch.einsum("sk,fsc->fkc", q["B"], self.X[q["P"]])
            b1, b2 = G[:, 1], G[:, 2]
            nrm = torch.linalg.cross(b1, b2)
            nn = nrm.norm(dim=1, keepdim=True)
            n = nrm / nn
            ez = torch.zeros_like(n)
            ez[:, 2] = 1.0
            j = ez - _dot(ez, n)[:, None] * n
            k = -torch.linalg.cross(n, j)
            j, k = nn.sqrt() * j / j.norm(dim=1, keepdim=True), nn.sqrt() * k / k.norm(dim=1, keepdim=True)
            g11, g12, g22 = _dot(b1, b1), _dot(b1, b2), _dot(b2, b2)
            det = g11 * g22 - g12 * g12
            co = lambda t: ((g22 * _dot(t, b1) - g12 * _dot(t, b2)) / det, (g11 * _dot(t, b2) - g12 * _dot(t, b1)) / det)  # noqa: E731
            q["R0"], q["R1"] = co(k), co(j)
            q["JxW"] = 0.5 * nn[:, 0]
            q["ref"] = self._rotate(q, G)
            A1, A2 = q["ref"][:2]
            c = torch.linalg.cross(A1, A2)
            q["L0"] = c.norm(dim=1)
            q["N0"] = c / q["L0"][:, None]
            f0, f1, f2 = _dot(A1, A1), _dot(A2, A2), _dot(A1, A2)
            s2 = 1 / (f0 * f1 - f2 * f2) ** 2
            e1, e2, nu, gg = g("e1"), g("e2"), g("nu"), g("g")
            w = 1 - nu * (e1 * nu / e2)
            q["H"] = (s2 * e1 * f1 * f1, s2 * e1 * (nu * f1 * f0 + (1 - nu) * f2 * f2), -s2 * e1 * f1 * f2,
                      s2 * e2 * f0 * f0, -s2 * e2 * f0 * f2,
                      s2 * gg * (w * f1 * f0 + w * (1 + nu) / (1 - nu) * f2 * f2))
            mass = (q["B"][:, 0].sum() * q["JxW"] * g("h"))[:, None] * q["B"][None, :, 0]
            M.index_add_(0, q["P"].reshape(-1), mass.reshape(-1))
            C.index_add_(0, q["P"].reshape(-1), (g("alpha")[:, None] * mass).reshape(-1))
            self.groups.append(q)
        self.M, self.C = M[:, None], C[:, None]

    @staticmethod
    def _rotate(q, G):
        (r00, r10), (r01, r11) = [[x[:, None] for x in r] for r in (q["R0"], q["R1"])]
        return (r00 * G[:, 1] + r10 * G[:, 2], r01 * G[:, 1] + r11 * G[:, 2],
                r00 * r00 * G[:, 3] + r10 * r10 * G[:, 4] + 2 * r00 * r10 * G[:, 5],
                r01 * r01 * G[:, 3] + r11 * r11 * G[:, 4] + 2 * r01 * r11 * G[:, 5],
                r00 * r01 * G[:, 3] + r10 * r11 * G[:, 4] + (r01 * r10 + r00 * r11) * G[:, 5])

    def forces(self, u, pressure, internal=True):
        """External pressure minus internal force per node; per-face measurement sums in self.meas."""
        f = torch.zeros(self.V, 3, **_F64)
        self.area = torch.zeros(self.F, **_F64)
        meas = torch.zeros(5, **_F64)
        x = torch.linalg.cross
        for q in self.groups:
            d1, d2, e1, e2, e3 = self._rotate(q, torch.einsum("sk,fsc->fkc", q["B"], u[q["P"]]))
            A1, A2, D1, D2, D3 = q["ref"]
            al = (_dot(A1, d1) + 0.5 * _dot(d1, d1), _dot(A2, d2) + 0.5 * _dot(d2, d2),
                  _dot(A1, d2) + _dot(d1, A2) + _dot(d1, d2))
            Dn = x(A1, d2) + x(d1, A2) + x(d1, d2)
            dL = 2 * q["L0"] * _dot(q["N0"], Dn) + _dot(Dn, Dn)
            jac = (q["L0"] ** 2 + dL).sqrt()
            dn = Dn / jac[:, None] - q["N0"] * (dL / ((q["L0"] + jac) * jac))[:, None]
            a3 = q["N0"] + dn
            a1, a2, v1, v2, v3 = A1 + d1, A2 + d2, D1 + e1, D2 + e2, D3 + e3
            be = (-(_dot(D1, dn) + _dot(e1, a3)), -(_dot(D2, dn) + _dot(e2, a3)), -2 * (_dot(D3, dn) + _dot(e3, a3)))
            H00, H01, H02, H11, H12, H22 = q["H"]
            mul = lambda s, t: (s * (H00 * t[0] + H01 * t[1] + H02 * t[2]), s * (H01 * t[0] + H11 * t[1] + H12 * t[2]),  # noqa: E731
                                s * (H02 * t[0] + H12 * t[1] + H22 * t[2]))
            on = 1.0 if internal else 0.0
            nf, mf = mul(on * q["K"], al), mul(on * q["D"], be)
            h = _dot(v1, a3), _dot(v2, a3), _dot(v3, a3)
            c = lambda s: s[:, None]  # noqa: E731
            Mv = c(mf[0]) * v1 + c(mf[1]) * v2 + 2 * c(mf[2]) * v3
            sm = mf[0] * h[0] + mf[1] * h[1] + 2 * mf[2] * h[2]
            Y1 = c(nf[0]) * a1 + c(nf[2]) * a2 + (x(Mv, a2) + c(sm) * x(a2, a3)) / c(jac)
            Y2 = c(nf[1]) * a2 + c(nf[2]) * a1 + (x(a1, Mv) + c(sm) * x(a3, a1)) / c(jac)
            (r00, r10), (r01, r11) = [[c(s) for s in r] for r in (q["R0"], q["R1"])]
            y11, y22, y12 = -c(mf[0]) * a3, -c(mf[1]) * a3, -2 * c(mf[2]) * a3
            Z = torch.stack([-pressure * c(q["ps"]) * a3, r00 * Y1 + r01 * Y2, r10 * Y1 + r11 * Y2,
                             r00 * r00 * y11 + r01 * r01 * y22 + r00 * r01 * y12,
                             r10 * r10 * y11 + r11 * r11 * y22 + r10 * r11 * y12,
                             2 * r00 * r10 * y11 + 2 * r01 * r11 * y22 + (r01 * r10 + r00 * r11) * y12], 1)
            Z = Z * q["JxW"][:, None, None]
            share = torch.einsum("sk,fkc->fsc", q["B"], Z)
            f.index_add_(0, q["P"].reshape(-1), -share.reshape(-1, 3))
            area = 0.5 * jac
            self.area[q["ids"]] = area
            g = _dot(a1, a1), _dot(a2, a2), _dot(a1, a2)
            det = g[0] * g[1] - g[2] * g[2]
            meas += torch.stack([(0.5 * q["JxW"] * sum(p * s for p, s in zip(nf, al))).sum(),
                                 (0.5 * q["JxW"] * sum(p * s for p, s in zip(mf, be))).sum(), area.sum(),
                                 (area * (h[0] * h[1] - h[2] * h[2]) / det).sum(),
                                 (area * 0.5 * (h[0] * g[1] + h[1] * g[0] - 2 * h[2] * g[2]) / det).sum()])
        self.meas = meas
        return f


_F64 = {"dtype": torch.float64, "device": _DEV}


def _friction(fn, n, v, vn, k, mu_s, mu_d, damping, stick, orig, cp, v_stop=0.03):
    """Slip-stick friction; returns force, energy, stick flags and spring origins."""
    vt = v - vn[:, None] * n
    av = vt.norm(dim=1)
    eps = 1e-8 * v_stop
    slow = av <= v_stop
    new = slow & ~stick
    pre = mu_d * fn / (k * (av + eps)) - damping
    orig = torch.where(new[:, None], cp - pre[:, None] * vt, orig)
    us = cp - orig
    us = us - _dot(us, n)[:, None] * n
    f = torch.where(slow[:, None], -k * us - damping * k * vt, torch.zeros_like(us))
    e = torch.where(slow, 0.5 * k * _dot(us, us), torch.zeros_like(av))
    slip = ~slow | (_dot(f, f) >= (mu_s * fn) ** 2)
    f = torch.where(slip[:, None], (-mu_d * fn / (av + eps))[:, None] * vt, f)
    zero = torch.zeros_like(orig)
    return f, torch.where(slip, torch.zeros_like(e), e), (stick | slow) & ~slip, torch.where(slip[:, None], zero, orig)


def _closest(P, Q):
    """Closest points of triangles P and Q (m x 3 x 3): squared distance, vector P to Q, barycentric coordinates."""
    m = len(P)
    best = torch.full((m,), math.inf, **_F64)
    dc, bp, bq = torch.zeros(m, 3, **_F64), torch.zeros(m, 3, **_F64), torch.zeros(m, 3, **_F64)

    def take(lp, lq):
        nonlocal best, dc, bp, bq
        d = (lq[:, :, None] * Q).sum(1) - (lp[:, :, None] * P).sum(1)
        d2 = _dot(d, d)
        w = d2 < best
        best = torch.where(w, d2, best)
        dc, bp, bq = (torch.where(w[:, None], new, old) for new, old in ((d, dc), (lp, bp), (lq, bq)))

    def on_edge(i, s):
        l = torch.zeros(m, 3, **_F64)
        l[:, i], l[:, (i + 1) % 3] = 1 - s, s
        return l

    for i in range(3):
        for j in range(3):
            d1, d2, r = P[:, (i + 1) % 3] - P[:, i], Q[:, (j + 1) % 3] - Q[:, j], P[:, i] - Q[:, j]
            a, e, f, c, b = _dot(d1, d1), _dot(d2, d2), _dot(d2, r), _dot(d1, r), _dot(d1, d2)
            den = a * e - b * b
            s = torch.where(den > 0, ((b * f - c * e) / den).clamp(0, 1), torch.zeros_like(a))
            t = ((b * s + f) / e).clamp(0, 1)
            s = ((b * t - c) / a).clamp(0, 1)
            take(on_edge(i, s), on_edge(j, t))
    for A, B, swap in ((P, Q, False), (Q, P, True)):
        for j in range(3):
            e1, e2, r = B[:, 1] - B[:, 0], B[:, 2] - B[:, 0], A[:, j] - B[:, 0]
            g11, g12, g22, r1, r2 = _dot(e1, e1), _dot(e1, e2), _dot(e2, e2), _dot(e1, r), _dot(e2, r)
            det = g11 * g22 - g12 * g12
            v, w = (g22 * r1 - g12 * r2) / det, (g11 * r2 - g12 * r1) / det
            ok = (v >= 0) & (w >= 0) & (v + w <= 1)  # otherwise an edge test holds the minimum
            lb = torch.where(ok[:, None], torch.stack([1 - v - w, v, w], 1), torch.tensor([1.0, 0, 0], **_F64))
            la = torch.zeros(m, 3, **_F64)
            la[:, j] = 1.0
            take(*((lb, la) if swap else (la, lb)))
    return best, dc, bp, bq


def _contact_pairs(E, p, h):
    """Face pairs of a folded shell that are not neighbours and lie within 1.3 h of each other."""
    tri = p[E.T]
    cen = tri.mean(1)
    rad = (tri - cen[:, None]).norm(dim=2).max()
    reach = 1.3 * h + 2 * rad
    out = []
    for k in range(0, E.F, 4096):
        near = torch.cdist(cen[k:k + 4096], cen, compute_mode="donot_use_mm_for_euclid_dist") < reach
        i, j = near.nonzero(as_tuple=True)
        i = i + k
        w = i < j
        i, j = i[w], j[w]
        shared = (E.T[i][:, :, None] == E.T[j][:, None, :]).any(2).any(1)
        i, j = i[~shared], j[~shared]
        for q in range(0, len(i), 1 << 20):
            s = slice(q, q + (1 << 20))
            d2 = _closest(tri[i[s]], tri[j[s]])[0]
            ref = _closest(E.X[E.T[i[s]]], E.X[E.T[j[s]]])[0]
            w = (d2 < (1.3 * h) ** 2) & (ref >= (1.4 * h) ** 2)
            out.append(torch.stack([i[s][w], j[s][w]], 1))
    return torch.cat(out)


def _self_contact(E, st, p, v, f):
    """Adds the self-contact forces at positions p (velocities v) to f; returns Eself, Efric, contacts."""
    m = E.m
    h, nu21 = float(m["h"][0]), float(m["e2"][0] * m["nu"][0] / m["e1"][0])
    e_avg, one = 0.5 * float(m["e1"][0] + m["e2"][0]), 1 - float(m["nu"][0]) * nu21
    t1, t2 = E.T[st["pairs"][:, 0]], E.T[st["pairs"][:, 1]]
    d2, dc, b1, b2 = _closest(p[t1], p[t2])
    d = d2.sqrt()
    on = d < h
    n = dc / d[:, None]
    stiff = 0.5 * e_avg / (one * h) * torch.minimum(E.area[st["pairs"][:, 0]], E.area[st["pairs"][:, 1]])
    dep = h - d
    fn = torch.where(on, stiff * dep * 0.5 * (1 + h / d), torch.zeros_like(d))
    es = torch.where(on, 0.5 * stiff * (0.5 * dep * dep - dep * h + h * h * torch.log(h / d)), torch.zeros_like(d))
    vr = (b2[:, :, None] * v[t2]).sum(1) - (b1[:, :, None] * v[t1]).sum(1)
    cp = (b1[:, :, None] * p[t1]).sum(1) + 0.5 * dc
    ff, ef, stick, orig = _friction(fn, n, vr, _dot(vr, n), e_avg * h / one, MU, MU, 0.0, st["stick"], st["orig"], cp)
    st["stick"], st["orig"] = stick & on, torch.where(on[:, None], orig, torch.zeros_like(orig))
    fc = torch.where(on[:, None], ff + fn[:, None] * n, torch.zeros_like(n))
    f.index_add_(0, t1.reshape(-1), (b1[:, :, None] * (-0.5 * fc)[:, None, :]).reshape(-1, 3))
    f.index_add_(0, t2.reshape(-1), (b2[:, :, None] * (0.5 * fc)[:, None, :]).reshape(-1, 3))
    return es.sum(), torch.where(on, ef, torch.zeros_like(ef)).sum(), int(on.sum())


def _cavity(E, st, p, v, f):
    """Adds the ellipsoidal cavity's forces to f; returns energy, friction energy, contacts."""
    c, m = _CAVITY, E.m
    h = float(m["h"][0])
    nu21 = float(m["e2"][0] * m["nu"][0] / m["e1"][0])
    e_avg, one = 0.5 * float(m["e1"][0] + m["e2"][0]), 1 - float(m["nu"][0]) * nu21
    R = torch.tensor(c["R"], **_F64) - 0.5 * h
    avg = R.mean()
    opd = ((p / R) ** 2).sum(1)
    near = opd > (1 - 0.1 * h / avg) ** 2
    depth = avg * (opd.sqrt() - 1)
    area, cnt = torch.zeros(E.V, **_F64), torch.zeros(E.V, **_F64)
    area.index_add_(0, E.T.reshape(-1), E.area.repeat_interleave(3))
    cnt.index_add_(0, E.T.reshape(-1), torch.ones(3 * E.F, **_F64))
    stiff = 0.5 * e_avg / (one * h) * area / cnt
    inside = near & (depth > 0)
    fn = torch.where(inside, stiff * depth, torch.zeros_like(depth))
    n = p / R ** 2
    n = n / n.norm(dim=1, keepdim=True)
    vn = _dot(v, n)
    ff, ef, stick, orig = _friction(fn, n, v, vn, e_avg * h / one, c["mu_s"], c["mu_d"], c["fric_damping"],
                                    (st["orig"] ** 2).sum(1) != 0, st["orig"], p)
    st["orig"] = torch.where(near[:, None], orig, torch.zeros_like(orig))
    f += torch.where(near[:, None], ff - (fn + c["damping"] * stiff * vn)[:, None] * n, torch.zeros_like(n))
    return torch.where(inside, 0.5 * stiff * depth ** 2, torch.zeros_like(depth)).sum(), \
        torch.where(near, ef, torch.zeros_like(ef)).sum(), int(inside.sum())


def _exact_network(d):
    P = [(_t(W), _t(b)) for W, b in d["params"]]
    X, T = _t(d["X"]), _t(d["T"])
    for W, b in P:
        W.requires_grad_(True)
        b.requires_grad_(True)
    Hh = X
    for k, (W, b) in enumerate(P):
        Hh = Hh @ W.T + b
        if k < len(P) - 1:
            Hh = torch.nn.functional.gelu(Hh)
    loss = ((Hh - T) ** 2).mean()
    loss.backward()
    return [np.array([loss.item()])] + [W.grad.cpu().numpy() for W, _ in P] + [b.grad.cpu().numpy() for _, b in P]


def exact(case, seed):
    kind = case["kind"]
    if kind == "folded" and case["contact"] == "smooth":
        return None  # a local search's end point: it has no value apart from the search
    d = _inputs(case, seed)
    if kind == "network":
        return _exact_network(d)
    E = _Exact(d)
    u, v = _t(d["u"]).reshape(-1, 3), _t(d["v"]).reshape(-1, 3)
    out = lambda x: x.reshape(-1).cpu().numpy()  # noqa: E731
    if kind == "forces":
        f = E.forces(u, float(d["table"][0]))
        return [out(f), out((f - E.C * v) / E.M), E.meas[:3].cpu().numpy()]
    a = torch.zeros_like(u)
    dt = E.dt
    beta, gamma = 0.25, 0.5
    st = {"orig": torch.zeros_like(u)}
    if kind == "folded":
        st["pairs"] = _contact_pairs(E, E.X + u, float(E.m["h"][0]))
        st["stick"] = torch.zeros(len(st["pairs"]), dtype=torch.bool, device=_DEV)
        st["orig"] = torch.zeros(len(st["pairs"]), 3, **_F64)
    extra, n_self, n_cav = [0.0, 0.0, 0.0], 0, 0  # Eself, Efric, Ecav
    for pr in d["table"]:
        up = u + dt * v + dt * dt * (0.5 - beta) * a
        vp = v + (1 - gamma) * dt * a
        f = E.forces(up, float(pr))
        if kind == "folded":
            extra[0], extra[1], n_self = _self_contact(E, st, E.X + up, v, f)
        if kind == "cavity":
            extra[2], extra[1], n_cav = _cavity(E, st, E.X + up, v, f)
        a = (f - E.C * vp) / E.M
        u, v = up + beta * dt * dt * a, vp + gamma * dt * a
    ekin = 0.5 * (v * v * E.M).sum()
    m = E.meas
    report = np.array([float(x) for x in (m[0], m[1], extra[0], extra[1], ekin, m[2], m[3], m[4], extra[2])])
    res = [out(u), out(v), out(a), report, np.array([len(d["table"]), n_self, n_cav], dtype=np.int64)]
    if kind == "relax":
        fi, fe = E.forces(u, float(d["table"][-1])), E.forces(u, float(d["table"][-1]), internal=False)
        k = len(d["mats"])
        tot = lambda x: torch.zeros(k, x.shape[1], **_F64).index_add_(0, E.node_shell, x)  # noqa: E731
        mass = tot(E.M)
        free = lambda x: x - E.M * (tot(x) / mass)[E.node_shell]  # noqa: E731
        sq = lambda x: tot((x * x).sum(1, keepdim=True))[:, 0]  # noqa: E731
        res.append((sq(free(fi)) / sq(free(fe))).sqrt().cpu().numpy())
    return res
