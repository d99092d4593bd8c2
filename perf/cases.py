"""Performance cases: the work that users of this package have it do, through its public entry points.

Every case is a dict of plain values.  `path` names the entry points it goes through:

  step       Solver.step(steps), state read into a page-locked buffer: the solver's main loop (explicit
             steps with a proximity update every ten), read back at the cadence of a monitoring program
  monitored  the same with device Monitoring set up: one row per step, drained after the call
  adaptive   Solver.step under the Adaptive_Euler scheme (two force evaluations an attempt, accept/reject)
  host       a drop-in host loop whose state lives in host memory: upload, one step, download
  batch      Batch.step over several independent samples of uneven size
  proximity  one step, contact pressures, Update_proximity on demand and the contact list it leaves
  mls        mls_shapes: shape functions of a sample's Gauss points, host arrays in and out

Two kinds of sample: "lattice" is the small plate-pressed square lattice of discs with 48 border and
100 interior nodes, whose contacts carry load from the first step; "packing" is the biaxial sample of
`grains` polydisperse discs, border nodes uniform in [border_lo, border_hi], five times as many interior
nodes, plates at 0.05 m/s and walls under confining pressure.  Samples start in motion: every grain has its
own velocity, spin and strain, so that internal forces act at once and grains collide later."""
import ctypes as C
import functools
import math

import numpy as np

from melody2d_b200 import abi
from melody2d_b200 import generator as g
from melody2d_b200 import solver as sv

GRADES = (32, 48, 64, 80, 96)          # border counts that have a disc template
ADAPTIVE = (2e-3, 0.2, 0.9)           # target error, smallest and largest ratio of successive steps


class _Templates(g.DiscTemplates):
    """Disc templates for a few border counts; the counts between them take the nearest."""

    @staticmethod
    def _grade(n):
        return min(GRADES, key=lambda c: abs(c - n))

    def grain(self, n_border, *a, **k):
        return super().grain(self._grade(n_border), *a, **k)

    def critical_dt(self, n_border, *a):
        return super().critical_dt(self._grade(n_border), *a)


@functools.lru_cache(maxsize=None)
def _templates():
    return _Templates(GRADES, workers=1)


def _case(name, path, sample, precision="fp64", material="elastic", steps=1, grains=16, border_lo=64, border_hi=64,
          samples=1, boundaries=False):
    return dict(name=name, path=path, sample=sample, precision=precision, material=material, steps=steps, grains=grains,
                border_lo=border_lo, border_hi=border_hi, samples=samples)


def listed():
    return [
        # one step of the smallest model and its monitored quantities: an interactive or coupled
        # program that looks at every step; launches and latency
        _case("lattice_one_step", "step", "lattice"),
        # the small reference workload: wall force and energies recorded along 100 steps
        _case("lattice_monitored", "monitored", "lattice", steps=100),
        # adaptive time step on a small model: two half-steps an attempt, errors read on the host
        _case("lattice_adaptive", "adaptive", "lattice", steps=20),
        # a small sample of the batched workload on its own: fewer bodies than SMs
        _case("packing50_fp64", "step", "packing", steps=100, grains=50, border_lo=32, border_hi=96),
        # rubber-like grains in the mixed form, about two bodies an SM
        _case("packing250_neohookean_mixed", "step", "packing", "mixed", "neohookean", steps=50, grains=250),
        # the large single sample in the plain FP64 form, and in the mixed form
        _case("packing700_fp64", "step", "packing", steps=50, grains=700),
        _case("packing700_mixed", "step", "packing", "mixed", steps=50, grains=700),
        # a slice of the batched workload: samples of uneven size in shared launches
        _case("batch8_mixed", "batch", "packing", "mixed", steps=50, grains=100, border_lo=32, border_hi=96, samples=8),
        # drop-in use: the host owns the state and hands it over at every step
        _case("host_packing200_fp64", "host", "packing", grains=200),
        _case("host_packing60_mixed", "host", "packing", "mixed", grains=60, border_lo=48, border_hi=80),
        # contact detection on demand with the contact quantities an analysis reads
        _case("proximity_packing400", "proximity", "packing", grains=400),
        # input generation of a 100-grain sample
        _case("mls_packing100", "mls", "packing", grains=100, border_lo=32, border_hi=96),
    ]


def draw(rng):
    def sized(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    lo = rng.randint(32, 96)
    hi = rng.randint(lo, 96)
    precision = rng.choice(["fp64", "mixed"])
    material = rng.choice(["elastic", "elastic", "elastic", "neohookean"])
    path = rng.choice(["step", "step", "step", "batch", "host", "proximity", "monitored", "adaptive", "mls"])
    c = _case("drawn", path, "packing", precision, material, 1, 50, lo, hi)
    del c["name"]
    if path == "step":
        c.update(grains=sized(8, 450), steps=sized(1, 50))
    elif path == "batch":
        c.update(grains=sized(10, 80), samples=rng.randint(2, 8), steps=sized(5, 50))
    elif path == "host":
        c.update(grains=sized(8, 200))
    elif path == "proximity":
        c.update(grains=sized(8, 400))
    elif path in ("monitored", "adaptive"):
        c.update(sample="lattice", grains=rng.choice([4, 6, 9, 12, 16, 20, 25]), steps=sized(5, 100), material="elastic",
                 border_lo=48, border_hi=48)
    else:
        c.update(grains=sized(4, 120), precision="fp64", material="elastic")
    return c


# ---- inputs -------------------------------------------------------------------------------------
# The geometry of a case (packing, nodes, shape functions) is that of its sizes; what the seed gives is
# the state the grains are in, as when one sample is loaded in different ways.
def _sides(n):
    ny = max(d for d in range(1, math.isqrt(n) + 1) if n % d == 0)
    return n // ny, ny


@functools.lru_cache(maxsize=16)
def _model(path, sample, grains, border_lo, border_hi, material, index):
    """The flattened sample, grains first, and its grains as generated."""
    if sample == "lattice":
        nx, ny = _sides(grains)
        sc = g.disc_lattice_scene(seed=index, nx=nx, ny=ny, pitch=2.05e-3, gap0=-1e-6)
    else:
        sc = g.batch_sample_scene(index, _templates(), grains=(grains, grains), border=(border_lo, border_hi))
    if material == "neohookean":
        sc.materials = [(name, 1 if name == "Grain" else t, p) for name, t, p in sc.materials]
    if path == "adaptive":
        sc.solver, sc.solver_params = 1, ADAPTIVE + tuple(sc.solver_params)[len(ADAPTIVE):]
    if path == "mls":
        return None, [b for b in sc.bodies if b.kind == "deformable"]
    return g.flatten(sc), None


def _models(case):
    path = case["path"] if case["path"] in ("adaptive", "mls") else ""
    # samples of a batch are uneven: between half and one and a half times the stated size
    n = case["samples"]
    return [_model(path, case["sample"], max(2, int(case["grains"] * (0.5 + (k + 0.5) / n))) if n > 1 else case["grains"],
                   case["border_lo"], case["border_hi"], case["material"], k) for k in range(n)]


def _flats(case, seed):
    """The case's models with the state that `seed` gives every grain: a velocity, a spin and a
    uniform strain (for the lattice, smaller ones: its contacts are closed already)."""
    out = []
    rng = np.random.default_rng(seed)
    scale = 1.0 if case["sample"] == "packing" else 0.05
    for f, _ in _models(case):
        f = dict(f)
        x0, st = f["node_x0"].reshape(-1, 2), f["node_state"].reshape(-1, 12).copy()
        ptr = f["body_node_ptr"]
        for b in range(len(f["body_type"])):
            if f["body_type"][b] == 0:
                s = slice(ptr[b], ptr[b + 1])
                rel = x0[s] - x0[s].mean(axis=0)
                up = rel @ rng.normal(0.0, 1e-4 * scale, (2, 2))
                spin = rng.normal(0.0, 10.0 * scale)
                vp = rng.normal(0.0, 0.1 * scale, 2) + spin * np.stack([-rel[:, 1], rel[:, 0]], axis=1)
                st[s, 0:2] = st[s, 6:8] = up       # linear fields: parameters and displacements agree
                st[s, 2:4] = st[s, 8:10] = vp
        f["node_state"] = st.reshape(-1)
        out.append(f)
    return out


def _mls_bodies(case, seed):
    """Points, nodes and support radii of every grain, scaled and turned as the seed says."""
    rng = np.random.default_rng(seed)
    out = []
    for b in _models(case)[0][1]:
        r, t = rng.uniform(0.8, 1.2), rng.uniform(0.0, 2 * math.pi)
        m = r * np.array([[math.cos(t), -math.sin(t)], [math.sin(t), math.cos(t)]])
        out.append((b.gp_xy @ m.T, b.nodes @ m.T, b.domain * r))
    return out


class _State:
    """Solvers and page-locked host buffers of one case."""

    def __init__(self, case, seed):
        self.case = case
        prec = 1 if case["precision"] == "mixed" else 0
        self.batch, self.solvers, self.host = None, [], []
        if case["path"] == "mls":
            self.bodies = _mls_bodies(case, seed)
            return
        flats = _flats(case, seed)
        self.solvers = [sv.Solver.from_flat(f, precision=prec, retain=False) for f in flats]
        self.host = [sv.PinnedArray(12 * s.nn) for s in self.solvers]
        for h, f in zip(self.host, flats):
            h.array[:] = f["node_state"]
        # nodes of the grains come first, those of the plates and walls after them
        self.split = [int(f["body_node_ptr"][int(np.argmax(f["body_type"] != 0))]) for f in flats]
        if case["path"] == "batch":
            self.batch = sv.Batch(precision=prec)
            for s in self.solvers:
                self.batch.admit(s)
        if case["path"] == "proximity":
            self.capacity = 32 * case["grains"]
            self.contacts = (abi.MelContact * self.capacity)()
        if case["path"] == "monitored":
            s = self.solvers[0]
            top, bottom = s.nb - 1, s.nb - 2
            # contact and driving force of both plates, travel of the upper one, kinetic energy, work
            # of the drive, and the velocity of the first grain's first node
            entries = [[4, 1, 2, top, -1], [4, 1, 2, bottom, -1], [4, 1, 4, top, -1], [1, 1, top, -1], [9, 0, -1],
                       [10, 3, -1], [2, 1, 0, 0]]
            s.monitor_setup(entries, energy=True, ring_rows=max(1000, case["steps"]))

    def read(self, k):
        """The node state of solver k in its page-locked buffer: grains, then plates and walls."""
        s, h = self.solvers[k], self.host[k].array
        sv._check(sv.lib().mel_get_node_state(s.h, sv._ptr(h)))
        a = h.reshape(-1, 12)
        return _parts(a[:self.split[k]], a[self.split[k]:])

    def read_contacts(self):
        """The contact list in the caller's buffer of fixed capacity, by field."""
        n = C.c_int()
        sv._check(sv.lib().mel_get_contacts(self.solvers[0].h, self.contacts, self.capacity, C.byref(n)))
        a = np.frombuffer(self.contacts, dtype=abi.CONTACT_DTYPE)
        return [n.value] + [np.ascontiguousarray(a[k]) for k in _CONTACT]

    def __del__(self):
        if self.batch is not None:
            self.batch.close()
        for s in self.solvers:
            s.close()
        for h in self.host:
            h.close()


_FIELDS = ("u", "v", "a", "u_param", "v_param", "a_param")


def _parts(grains, frame):
    """Kinematic fields of the grains' nodes, by field, and of the rigid frame's nodes."""
    out = {name: grains[:, 2 * i:2 * i + 2] for i, name in enumerate(_FIELDS)}
    out["frame"] = frame
    return out


def prepare(case, seed):
    return _State(case, seed)


def run(state):
    case, path = state.case, state.case["path"]
    if path == "mls":
        return _joined(sv.mls_shapes(state.bodies))
    s = state.solvers[0]
    if path == "batch":
        state.batch.step(case["steps"])
        return [state.read(k) for k in range(len(state.solvers))]
    if path == "host":
        sv._check(sv.lib().mel_set_node_state(s.h, sv._ptr(state.host[0].array)))
        s.step(1)
        return state.read(0)
    if path == "proximity":
        s.step(1, proximity=False)
        p = s.contact_pressures()
        s.update_proximity()
        return {"state": state.read(0), "pressures": p, "contacts": state.read_contacts()}
    s.step(case["steps"])
    if path == "monitored":
        return {"rows": np.stack(s.monitor_rows()), "state": state.read(0)}
    out = {"state": state.read(0)}
    if path == "step" and case["steps"] == 1:
        m = s.monitor()
        out["monitor"] = [m.kinetic_energy, *m.mean_displacement, *m.rigid_force, *m.rigid_dirichlet, m.active_contacts]
    return out


_CONTACT = ("bodyS", "nodeS", "bodyM", "segmentM", "gapn", "gapt", "xsi", "fx", "fy")


def _joined(csr):
    """The shape functions of all bodies, each column in one array."""
    return [np.concatenate([np.asarray(b[i]) for b in csr]) for i in range(5)]


# ---- what a pass cannot do without ----------------------------------------------------------------
def _disc(border, interior):
    """Nodes, Gauss points, their support entries and the nodes' support entries of one disc."""
    n = border + interior
    points = 3 * (2 * n - border - 2)
    return n, points, 15 * points, 13 * n


def work(case):
    if case["sample"] == "lattice":
        n, p, e, ne = _disc(48, 100)
    else:
        b = (case["border_lo"] + case["border_hi"]) / 2.0
        n, p, e, ne = _disc(b, 5 * b)
    discs = case["grains"] * case["samples"]
    if case["path"] == "mls":
        # points and nodes in, row pointers, index and three columns out; about 60 operations an entry
        return {"bytes": discs * (16.0 * p + 24.0 * n + 8.0 * p + 28.0 * e), "flops": discs * 60.0 * e}
    pair = 16.0 if case["precision"] == "fp64" else 8.0
    # per force evaluation: derivative pairs and node index of every entry, point weights, node
    # supports, and the node state read (x0, masses, parameters) and written
    step = discs * (e * (pair + 2.0) + 8.0 * p + 10.0 * ne + (80.0 + 112.0) * n)
    flops = discs * (18.0 * e + 12.0 * ne)
    evals = case["steps"] * (2 if case["path"] == "adaptive" else 1)
    read = discs * 96.0 * n * (2 if case["path"] == "host" else 1)
    return {"bytes": evals * step + read, "flops": evals * flops}


# ---- values in 64 bits, by plain numpy ----------------------------------------------------------------
def _exact_host(case, seed):
    """One explicit step of the grains, none of them in contact yet: internal forces of every Gauss
    point, Newton, Euler, and the kinematics through the nodes' shape functions."""
    if case["material"] == "neohookean":
        return None
    f = _flats(case, seed)[0]
    ng = int(np.argmax(f["body_type"] != 0))
    n = int(f["body_node_ptr"][ng])
    node0 = f["body_node_ptr"][:ng]
    gp0 = f["body_gp_ptr"][:ng + 1]
    P = int(gp0[-1])
    counts = np.diff(f["gp_sup_ptr"][:P + 1])
    E = int(f["gp_sup_ptr"][P])
    row = np.repeat(np.arange(P), counts)
    col = f["gp_sup_idx"][:E] + np.repeat(np.repeat(node0, np.diff(gp0)), counts)
    dx, dy = f["gp_dNdx"][:E], f["gp_dNdy"][:E]
    st = f["node_state"].reshape(-1, 12)[:n]
    up, vp = st[:, 6:8], st[:, 8:10]
    total = lambda v: np.bincount(row, weights=v, minlength=P)  # noqa: E731
    c0 = f["gp_weight"][:P] * f["gp_jacobian"][:P]
    young, nu = 1e8, 0.3
    mu, lam = young / (2 * (1 + nu)), young * nu / ((1 + nu) * (1 - 2 * nu))
    e11, e22 = total(dx * up[col, 0]), total(dy * up[col, 1])
    e12 = 0.5 * total(dx * up[col, 1] + dy * up[col, 0])
    s33 = lam * (e11 + e22)
    s11, s22, s12 = s33 + 2 * mu * e11, s33 + 2 * mu * e22, 2 * mu * e12
    fx = -np.bincount(col, weights=(c0[row] * (dx * s11[row] + dy * s12[row])), minlength=n)
    fy = -np.bincount(col, weights=(c0[row] * (dy * s22[row] + dx * s12[row])), minlength=n)
    force = np.stack([fx, fy], axis=1)
    dt = float(f["dt"])
    ap = force * f["node_inv_mass"].reshape(-1, 2)[:n]
    vp = vp + dt * ap
    up = up + dt * vp
    ptr = f["node_sup_ptr"][:n + 1]
    nrow = np.repeat(np.arange(n), np.diff(ptr))
    body_of = np.repeat(node0, np.diff(f["body_node_ptr"][:ng + 1]))
    ncol = f["node_sup_idx"][:ptr[-1]] + body_of[nrow]
    N = f["node_sup_N"][:ptr[-1]]
    u, v, a = (np.stack([np.bincount(nrow, weights=N * w[ncol, k], minlength=n) for k in (0, 1)], axis=1) for w in (up, vp, ap))
    return {"u": u, "v": v, "a": a, "u_param": up, "v_param": vp, "a_param": ap, "frame": None}


def _exact_mls(case, seed):
    """Linear moving least squares with the cubic-spline weight, point-centred and scaled by radius."""
    cols = [[], [], [], [], []]
    for pts, nodes, radii in _mls_bodies(case, seed):
        r = float(radii[0])
        d = (pts[:, None, :] - nodes[None, :, :]) / r
        q2 = (d * d).sum(axis=2)
        diff = pts[:, None, :] - nodes[None, :, :]
        inside = (diff * diff).sum(axis=2) - radii[None, :] ** 2 < 0.0
        pi, ni = np.nonzero(inside)
        counts = inside.sum(axis=1)
        x, y, q = d[pi, ni, 0], d[pi, ni, 1], np.sqrt(q2[pi, ni])
        inner = q <= 0.5
        w = np.where(inner, 2.0 / 3.0 - 4 * q ** 2 + 4 * q ** 3, 4.0 / 3.0 * (1 - q) ** 3)
        k = np.where(inner, -8.0 + 12.0 * q, -4.0 * (1 - q) ** 2 / np.where(inner, 1.0, q))   # w'(q) / q
        wx, wy = k * x, k * y
        P = len(pts)
        basis = [np.ones_like(x), -x, -y]

        def moments(v):
            m = np.empty((P, 3, 3))
            for i in range(3):
                for j in range(3):
                    m[:, i, j] = np.bincount(pi, weights=v * basis[i] * basis[j], minlength=P)
            return m

        A, Ax, Ay = moments(w), moments(wx), moments(wy)
        # the basis (1, X - x, Y - y) moves with the point x: shape functions do not depend on its
        # origin, so differentiate as if it stood still at this point
        e = np.zeros((P, 3, 1))
        e[:, 0] = 1.0
        g1 = np.linalg.solve(A, e)
        ex, ey = np.zeros((P, 3, 1)), np.zeros((P, 3, 1))
        ex[:, 1], ey[:, 2] = 1.0, 1.0
        g2 = np.linalg.solve(A, ex - Ax @ g1)
        g3 = np.linalg.solve(A, ey - Ay @ g1)
        at = lambda v: sum(v[pi, i, 0] * basis[i] for i in range(3))  # noqa: E731
        p1 = at(g1)
        cols[0].append(np.concatenate([[0], np.cumsum(counts)]))
        cols[1].append(ni)
        cols[2].append(p1 * w)
        cols[3].append((at(g2) * w + p1 * wx) / r)
        cols[4].append((at(g3) * w + p1 * wy) / r)
    return cols


def exact(case, seed):
    if case["path"] == "host":
        return _exact_host(case, seed)
    if case["path"] == "mls":
        return [np.concatenate(c) for c in _exact_mls(case, seed)]
    return None     # many steps with contact: no short closed restatement
