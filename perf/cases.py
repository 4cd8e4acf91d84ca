"""The workloads this framework is timed on, through its public entry points.

A pass is what a program does with the library: copy a state from pinned host
memory into a Domain, advance it, and copy the new state back (or reset and
run an ensemble, take a gradient, or compute nodal forces on device arrays).
`exact` advances the same inputs with a plain float64 torch restatement of the
method, which shares no code with the package.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("lulesh.jl_gb300"))
import lulesh_gb300 as L  # noqa: E402

STATE = ("x", "y", "z", "xd", "yd", "zd", "e", "p", "q", "v", "ss")
NODE = STATE[:6]
EDGE = 1.125  # the Sedov cube's edge
ENERGY = 3.948746e7 * (EDGE / 45) ** 3  # the deposit times the origin element's mass, the same on every mesh


# --- the cases ----------------------------------------------------------------

def listed():
    return [
        # the CI-sized mesh stepped by the host, one call per cycle: launches and latency
        {"name": "steps_8", "kind": "steps", "nx": 8, "cycles": 50, "mode": 0},
        # the reference's default mesh and iteration count, its own loop
        {"name": "steps_45", "kind": "steps", "nx": 45, "cycles": 10, "mode": 0},
        # the reference's CPU-runnable mesh on the device loop, LULESH 2.0 method
        {"name": "run_30", "kind": "run", "nx": 30, "cycles": 100, "mode": 7},
        # an odd size between the configured ones
        {"name": "run_77", "kind": "run", "nx": 77, "cycles": 20, "mode": 0},
        # the headline throughput mesh
        {"name": "run_150", "kind": "run", "nx": 150, "cycles": 20, "mode": 0},
        # the largest configured mesh, unbalanced regions with repeated EOS work
        {"name": "regions_256", "kind": "run", "nx": 256, "cycles": 4, "mode": 0, "reps": True, "balance": 4, "cost": 2},
        # the multi-rank decomposition as blocks, stepped with every Domain array kept
        {"name": "blocks_2x25", "kind": "steps", "nx": 25, "cycles": 10, "mode": 7, "blocks": 2, "aux": True},
        # a handful of small problems advanced together
        {"name": "ensemble_24_small", "kind": "ensemble", "n": 24, "lo": 4, "hi": 20, "pick": 5, "cycles": 60, "mode": 0},
        # a parameter study over the configured range of mesh sizes
        {"name": "ensemble_64", "kind": "ensemble", "n": 64, "lo": 16, "hi": 64, "pick": 196, "cycles": 30, "mode": 0},
        # the gradient of a short run of a small mesh
        {"name": "adjoint_15", "kind": "adjoint", "nx": 15, "cycles": 24, "mode": 7, "every": 7},
        # the configured gradient's mesh and checkpoint spacing
        {"name": "adjoint_48", "kind": "adjoint", "nx": 48, "cycles": 40, "mode": 0, "every": 20},
        # nodal forces on a caller's own device arrays
        {"name": "force_27", "kind": "force", "nx": 27, "mode": 0},
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49))))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "run", "run", "run", "blocks", "ensemble", "ensemble", "adjoint", "adjoint", "force"])
    mode = rng.choice([0, 0, 7])
    if kind == "steps":
        return {"kind": "steps", "nx": _log_int(rng, 2, 96), "cycles": rng.randint(5, 50), "mode": mode,
                "aux": rng.random() < 0.3, "reps": rng.random() < 0.2, "balance": 2, "cost": 2}
    if kind == "run":
        nx = _log_int(rng, 6, 200)
        return {"kind": "run", "nx": nx, "cycles": max(4, min(100, int(2e7 / nx ** 3))), "mode": mode,
                "reps": rng.random() < 0.2, "balance": rng.randint(1, 4), "cost": rng.randint(1, 2)}
    if kind == "blocks":
        tp = rng.choice([2, 3])
        return {"kind": "steps", "nx": _log_int(rng, 3, 60 // tp), "cycles": rng.randint(4, 20), "mode": mode, "blocks": tp,
                "aux": rng.random() < 0.5}
    if kind == "ensemble":
        lo = _log_int(rng, 2, 24)
        return {"kind": "ensemble", "n": _log_int(rng, 2, 48), "lo": lo, "hi": lo + rng.randint(2, 36), "pick": rng.randint(1, 999),
                "cycles": rng.randint(10, 40), "mode": mode}
    if kind == "adjoint":
        return {"kind": "adjoint", "nx": _log_int(rng, 4, 48), "cycles": rng.randint(6, 40), "mode": mode, "every": rng.randint(4, 20)}
    return {"kind": "force", "nx": _log_int(rng, 2, 32), "mode": mode}


# --- inputs -------------------------------------------------------------------

def _mesh(nx, device="cpu"):
    """Undeformed node positions [3, N] and the corner list [8, E]."""
    c = EDGE * torch.arange(nx + 1, dtype=torch.float64, device=device) / nx
    z, y, x = torch.meshgrid(c, c, c, indexing="ij")
    en = nx + 1
    i = torch.arange(nx, device=device)
    k, j, i = torch.meshgrid(i, i, i, indexing="ij")
    n0 = (k * en * en + j * en + i).reshape(-1)
    off = [0, 1, en + 1, en, en * en, en * en + 1, en * en + en + 1, en * en + en]
    return torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)]), torch.stack([n0 + o for o in off])


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _blast(nx, seed):
    """A Sedov blast part of the way through the mesh, with seeded radius,
    energy, hourglass coefficient and smooth asymmetric perturbations: the
    state fields as host arrays and the scalars a restarted program sets."""
    r = np.random.default_rng(seed)
    dev = _device()
    X, nl = _mesh(nx, dev)
    rs, amp, hg = r.uniform(0.35, 0.7), r.uniform(0.5, 2.0), r.uniform(2.0, 4.0)
    wave, phase = torch.as_tensor(r.uniform(1, 7, (3, 3)), device=dev), torch.as_tensor(r.uniform(0, 6.28, (3, 1)), device=dev)

    def ripple(P):
        return torch.cos(wave @ P + phase)

    rad = X.square().sum(0).sqrt()
    s = rad / rs
    energy = ENERGY * amp
    speed = 0.4 * rs / math.sqrt((rs / 1.15) ** 5 / (8 * energy))  # the shock's speed over the blast's age
    # displaced outwards inside the shock, smoothly to nothing outside; planes through the origin stay planes
    P = X * (1 + 0.12 * torch.exp(-(s ** 4)) * (1 + 0.05 * ripple(X)))
    vel = X / rs * (0.75 * speed * torch.exp(-(s ** 6)) + 1e-3 * speed) * (1 + 0.1 * ripple(2 * X))
    C, C0 = P[:, nl], X[:, nl]
    v = _volume(*_triple(C)) / _volume(*_triple(C0))
    mid = C0.mean(1)
    se = mid.square().sum(0).sqrt() / rs
    noise = torch.as_tensor(r.random(nl.shape[1]), device=dev)
    e = energy / (rs ** 3 * 0.52) * (0.3 + 1.5 * torch.exp(-6 * se)) * torch.exp(-(se ** 8)) * (1 + 0.05 * noise) + 1e-3 * noise
    p = 2.0 / 3.0 * e / v
    q = 0.4 * p * torch.exp(-(((se - 0.95) / 0.08) ** 2))
    ss = (10.0 / 9.0 * e).sqrt()
    fields = dict(zip(STATE, (*P, *vel, e, p, q, v, ss)))
    h = EDGE / nx
    dt = 0.05 * h / (speed + float(ss.max()))
    return {k: f.cpu().numpy() for k, f in fields.items()}, {
        "time": 1e-3, "deltatime": dt, "dtcourant": 1e20, "dthydro": 1e20, "cycle": 0, "hgcoef": hg}


def _pinned(a):
    t = torch.from_numpy(np.ascontiguousarray(a))
    return t.pin_memory().numpy() if torch.cuda.is_available() else t.numpy()


def _block_ids(nx, tp):
    """Whole-mesh element and node ids of the packed blocks, in rank order."""
    el, no = [], []
    m = nx * tp
    for rank in range(tp ** 3):
        c, r, p = rank % tp, rank // tp % tp, rank // (tp * tp)
        for ids, n, w in ((el, nx, m), (no, nx + 1, m + 1)):
            k, j, i = np.meshgrid(p * nx + np.arange(n), r * nx + np.arange(n), c * nx + np.arange(n), indexing="ij")
            ids.append((k * w * w + j * w + i).reshape(-1))
    return np.concatenate(el), np.concatenate(no)


def _instances(case, seed):
    """The case's mesh sizes with seeded energies and hourglass coefficients."""
    r = np.random.default_rng(seed)
    spec = L.sedov_instances(seed=case["pick"], n=case["n"], nx_min=case["lo"], nx_max=case["hi"])
    for s in spec:
        s["einit"] = 3.948746e7 * (s["nx"] / 45.0) ** 3 * math.exp(r.uniform(math.log(0.5), math.log(2.0)))
        s["hgcoef"] = float(r.uniform(2.0, 4.0))
    return spec


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        return {"case": case, "ens": L.Ensemble(_instances(case, seed), mode=case["mode"])}
    nx, tp = case["nx"], case.get("blocks", 1)
    fields, scalars = _blast(nx * tp, seed)
    if kind == "force":
        return _prepare_force(case, fields, scalars)
    if tp > 1:
        eg, ng = _block_ids(nx, tp)
        fields = {k: f[ng if k in NODE else eg] for k, f in fields.items()}
    dom = L.Domain(L.LuleshProblem(nx=nx, nr=11, balance=case.get("balance", 1), cost=case.get("cost", 1), mode=case["mode"],
                                   region_reps=case.get("reps", False), keep_aux=case.get("aux", False), blocks_per_edge=tp))
    state = {"case": case, "dom": dom, "scalars": scalars, "in": {k: _pinned(f) for k, f in fields.items()}}
    if kind == "adjoint":
        state["adj"] = L.Adjoint(dom, radius=0.3, checkpoint_every=case["every"])
    else:
        state["out"] = {k: _pinned(np.empty_like(f)) for k, f in fields.items()}
    return state


def _prepare_force(case, fields, scalars):
    nx = case["nx"]
    X, nl = _mesh(nx, "cuda")
    E, N = nl.shape[1], X.shape[1]
    node = nl.t().reshape(-1)  # element-major
    order = torch.sort(node, stable=True).indices
    count = torch.bincount(node, minlength=N)
    volo = _volume(*_triple(X[:, nl]))
    dev = {k: torch.from_numpy(fields[k]).cuda() for k in STATE if k != "e"}
    dev |= {"volo": volo, "elemMass": volo.clone(), "nodelist": node.contiguous(), "nodeElemCount": count,
            "nodeElemStart": torch.cumsum(count, 0) - count, "nodeElemCornerList": order + 1}
    dev |= {k: torch.zeros(N, dtype=torch.float64, device="cuda") for k in ("fx", "fy", "fz")}
    args = L.ForceArgs(num_elem=E, num_node=N, hgcoef=scalars["hgcoef"], mode=case["mode"])
    for k, t in dev.items():
        setattr(args, k, t.data_ptr())
    fn = L.load_library().lulesh_calc_force_for_nodes_static
    fn.argtypes = [ctypes.POINTER(L.ForceArgs), ctypes.c_void_p, ctypes.POINTER(ctypes.c_int32)]
    fn.restype = ctypes.c_int
    return {"case": case, "fn": fn, "args": args, "dev": dev}


# --- a pass -------------------------------------------------------------------

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "force":
        site = ctypes.c_int32()
        rc = state["fn"](ctypes.byref(state["args"]), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.byref(site))
        if rc:
            raise RuntimeError("force status %d at site %d" % (rc, site.value))
        return {k: state["dev"][k] for k in ("fx", "fy", "fz")}
    if kind == "ensemble":
        ens = state["ens"]
        ens.reset()
        ens.run(case["cycles"])
        out = {k: np.concatenate([ens.field(i, k) for i in range(case["n"])]) for k in ("e", "x")}
        out["time"] = np.array([ens.scalars(i)["time"] for i in range(case["n"])])
        return out
    dom = state["dom"]
    for k, f in state["in"].items():
        dom.set_field(k, f)
    for k, s in state["scalars"].items():
        setattr(dom, k, s)
    if kind == "adjoint":
        adj = state["adj"]
        out = {"loss": adj.gradient(case["cycles"]), "hgcoef": adj.result.grad_hgcoef}
        out |= {k: adj.grad(k) for k in STATE}
        return out
    if kind == "steps":
        while dom.time < dom.stoptime:
            L.timeIncrement(dom)
            L.lagrangeLeapFrog(dom)
            if dom.cycle >= case["cycles"]:
                break
    else:
        L.run(dom, case["cycles"])
    out = {k: dom.field(k, out=f) for k, f in state["out"].items()}
    out["time"] = dom.time
    return out


def work(case):
    """Per zone and cycle: the FP64 operations of the method's own formulas
    (about 1,500) and each state field read and written once, with the masses,
    volumes and connectivity read; a gradient is about four such steps."""
    if case["kind"] == "ensemble":
        zones = sum(s["nx"] ** 3 for s in _instances(case, 0))
    else:
        zones = (case["nx"] * case.get("blocks", 1)) ** 3
    if case["kind"] == "force":
        return {"bytes": 8.0 * zones * (6 + 6 + 8 + 8 + 3 + 2), "flops": 800.0 * zones}
    steps = float(zones) * case["cycles"] * (4 if case["kind"] == "adjoint" else 1)
    return {"bytes": 519.0 * steps + 8.0 * 2 * 11 * zones, "flops": 1500.0 * steps}


# --- the method in plain float64 torch ----------------------------------------

def _triple(C):
    """The three triple products of 12 * volume: U, V, W of corner positions C [3, 8, E]."""
    def d(a, b):
        return C[:, a] - C[:, b]
    U = (d(3, 1) + d(7, 2), d(4, 3) + d(5, 7), d(1, 4) + d(2, 5))
    V = (d(6, 3), d(6, 4), d(6, 1))
    W = (d(2, 0), d(7, 0), d(5, 0))
    return U, V, W


def _cross(a, b):
    return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]])


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _volume(U, V, W):
    return sum(_dot(u, _cross(v, w)) for u, v, w in zip(U, V, W)) / 12.0


def _columns(C):
    """xi, eta, zeta sums of corner values C [3, 8, E] (8 times the Jacobian's columns)."""
    xi = C[:, 1] + C[:, 2] + C[:, 5] + C[:, 6] - C[:, 0] - C[:, 3] - C[:, 4] - C[:, 7]
    eta = C[:, 2] + C[:, 3] + C[:, 6] + C[:, 7] - C[:, 0] - C[:, 1] - C[:, 4] - C[:, 5]
    zeta = C[:, 4] + C[:, 5] + C[:, 6] + C[:, 7] - C[:, 0] - C[:, 1] - C[:, 2] - C[:, 3]
    return xi, eta, zeta


_FACES = ((0, 1, 2, 3), (0, 4, 5, 1), (1, 5, 6, 2), (2, 6, 7, 3), (3, 7, 4, 0), (4, 7, 6, 5))
_GAMMA = ((1, 1, -1, -1, -1, -1, 1, 1), (1, -1, -1, 1, -1, 1, 1, -1), (1, -1, 1, -1, 1, -1, 1, -1), (-1, 1, -1, 1, 1, -1, 1, -1))


def _face_normals(C):
    """Area vectors of the six faces, pointing inwards."""
    return [_cross(C[:, c] - C[:, a], C[:, d] - C[:, b]) / -2.0 for a, b, c, d in _FACES]


def _cut(x, c):
    return torch.where(x.abs() < c, torch.zeros_like(x), x)


class _Sedov:
    """One problem's constants and its cycle: state dict in, state dict out."""

    def __init__(self, nx, mode, device):
        self.nx, self.mode, self.device = nx, mode, device
        self.X, self.nl = _mesh(nx, device)
        self.volo = _volume(*_triple(self.X[:, self.nl]))
        N = self.X.shape[1]
        self.mass = torch.zeros(N, dtype=torch.float64, device=device)
        for c in range(8):
            self.mass.index_add_(0, self.nl[c], self.volo / 8.0)
        self.fixed = [self.X[k] == 0 for k in range(3)]

    def forces(self, s):
        mode, C, vel = self.mode, torch.stack([s["x"], s["y"], s["z"]])[:, self.nl], torch.stack([s["xd"], s["yd"], s["zd"]])[:, self.nl]
        normal = _face_normals(C)
        B = [sum(normal[f] for f in range(6) if n in _FACES[f]) / 4.0 for n in range(8)]
        if not mode & 1:  # the reference's node 0 takes the fifth face's y area twice and no z area
            skew = torch.zeros_like(B[0])
            skew[1] = 1
            skew = normal[4] / 4.0 * skew
            lack = torch.zeros_like(B[0])
            lack[2] = 1
            B[0] = B[0] + skew - lack * normal[4] / 4.0
        press = s["p"] + s["q"]
        U, V, W = _triple(C)
        gu = [_cross(v, w) for v, w in zip(V, W)]
        gv = [_cross(w, u) for w, u in zip(W, U)]
        gw = [_cross(u, v) for u, v in zip(U, V)]
        D = [-(gw[0] + gw[1] + gw[2]), gu[2] - gu[0] - gv[2], gu[2] - gu[0] + gw[0], gu[0] - gu[1] - gv[0],
             gu[1] - gu[2] - gv[1], gu[1] - gu[2] + gw[2], gv[0] + gv[1] + gv[2], gu[0] - gu[1] + gw[1]]
        if not mode & 2:  # the reference exchanges the derivatives of corners 1 and 3
            D[1], D[3] = D[3], D[1]
        determ = self.volo * s["v"]
        coef = -s["hgcoef"] * 0.01 * s["ss"] * self.volo / determ ** (1.0 / 3.0)
        F = [press * B[n] for n in range(8)]
        for g in _GAMMA:
            hx = sum(g[n] * C[:, n] for n in range(8)) / (12.0 * determ)
            shape = [g[n] - _dot(D[n], hx) for n in range(8)]
            h = coef * sum(shape[n] * vel[:, n] for n in range(8))
            F = [F[n] + shape[n] * h for n in range(8)]
        out = torch.zeros_like(self.X)
        for n in range(8):
            out = out.index_add(1, self.nl[n], F[n])
        return out

    def step(self, s):
        nx, mode = self.nx, self.mode
        # time step control
        t, dt, cycle = s["time"], s["deltatime"], s["cycle"]
        target = 1e-2 - t
        if cycle != 0:
            new = s["dtcourant"] / 2.0
            if float(s["dthydro"]) < float(new):
                new = s["dthydro"] * 2.0 / 3.0
            ratio = float(new) / float(dt)
            if ratio >= 1.0:
                new = dt if ratio < 1.1 else dt * 1.2 if ratio > 1.2 else new
            dt = new if float(new) < 1e-2 else torch.full_like(new, 1e-2)
        if float(dt) < float(target) < 4.0 * float(dt) / 3.0:
            target = 2.0 * dt / 3.0
        if float(target) < float(dt):
            dt = target
        o = {"time": t + dt, "deltatime": dt, "cycle": cycle + 1, "hgcoef": s["hgcoef"]}
        # nodes
        acc = self.forces(s) / self.mass
        for k, (a, b) in enumerate((("xd", "x"), ("yd", "y"), ("zd", "z"))):
            ak = torch.where(self.fixed[k], torch.zeros_like(acc[k]), acc[k])
            o[a] = _cut(s[a] + ak * dt, 1e-7)
            o[b] = s[b] + o[a] * dt
        # elements
        C, vel = torch.stack([o["x"], o["y"], o["z"]])[:, self.nl], torch.stack([o["xd"], o["yd"], o["zd"]])[:, self.nl]
        vol = _volume(*_triple(C))
        vnew = vol / self.volo
        delv = vnew - s["v"]
        normal = _face_normals(C)
        best = torch.zeros_like(vol)
        for f in (0, 5, 1, 2, 3, 4):
            area = 16.0 * _dot(normal[f], normal[f])
            best = torch.where(area > best, area, best)
        arealg = 4.0 * vol / best.sqrt()
        vw = _columns(vel)
        half = _columns(C - 0.5 * dt * vel)
        cof = (_cross(half[1], half[2]), _cross(half[2], half[0]), _cross(half[0], half[1]))
        vdov = sum(_dot(c, w) for c, w in zip(cof, vw)) / _dot(half[0], cof[0])
        w = _columns(C)
        volume = self.volo * vnew
        A = (_cross(w[1], w[2]), _cross(w[2], w[0]), _cross(w[0], w[1]))
        delx = [16.0 * volume / (_dot(a, a) + 256e-36).sqrt() for a in A]
        dv = [_dot(a, u) / (64.0 * volume + 64e-36) for a, u in zip(A, vw)]
        phi = []
        for d in range(3):
            g = dv[d].reshape(nx, nx, nx)
            axis = 2 - d
            first, last = g.narrow(axis, 0, 1), torch.zeros_like(g.narrow(axis, 0, 1))
            dm = torch.cat([first, g.narrow(axis, 0, nx - 1)], axis).reshape(-1)
            rest = g.narrow(axis, 1, nx - 1)
            if d == 0 and not mode & 4:  # the reference's xi-plus neighbour is the element itself
                rest = g.narrow(axis, 0, nx - 1)
            dp = torch.cat([rest, last], axis).reshape(-1)
            norm = 1.0 / (dv[d] + 1e-36)
            dm, dp = dm * norm, dp * norm
            f = 0.5 * (dm + dp)
            f = torch.where(2.0 * dm < f, 2.0 * dm, f)
            f = torch.where(2.0 * dp < f, 2.0 * dp, f)
            f = torch.where(f < 0.0, torch.zeros_like(f), f)
            phi.append(torch.where(f > 1.0, torch.ones_like(f), f))
        zero = torch.zeros_like(vnew)
        dx = [torch.where(a * b > 0.0, zero, a * b) for a, b in zip(dv, delx)]
        rho = 1.0 / vnew
        ql = torch.where(vdov > 0.0, zero, -0.5 * rho * sum(x * (1.0 - f) for x, f in zip(dx, phi)))
        qq = torch.where(vdov > 0.0, zero, 2.0 / 3.0 * rho * sum(x * x * (1.0 - f * f) for x, f in zip(dx, phi)))
        # energy, pressure, viscosity
        c1 = 2.0 / 3.0
        b, bh = c1 / vnew, c1 / (vnew - 0.5 * delv)
        squeezed = delv <= 0.0

        def pressure(e, f):
            pn = _cut(f * e, 1e-7)
            return torch.where(pn < 0.0, zero, pn)

        def root(c):
            tiny = c <= 0.111111e-36
            return torch.where(tiny, torch.full_like(c, 0.333333e-18), torch.where(tiny, torch.ones_like(c), c).sqrt())

        pq = s["p"] + s["q"]
        e = s["e"] - 0.5 * delv * pq
        ph = pressure(e, bh)
        q = torch.where(squeezed, root(c1 * e + (vnew - 0.5 * delv) ** 2 * bh * ph) * ql + qq, zero)
        sh = ph + q
        e = _cut(e + 0.5 * delv * (3.0 * pq - 4.0 * sh), 1e-7)
        p = pressure(e, b)
        q = torch.where(squeezed, root(c1 * e + vnew * vnew * b * p) * ql + qq, zero)
        e = _cut(e - (7.0 * pq - 8.0 * sh + p + q) * delv / 6.0, 1e-7)
        p = pressure(e, b)
        o["ss"] = root(c1 * e + vnew * vnew * b * p)
        o["q"] = torch.where(squeezed, _cut(o["ss"] * ql + qq, 1e-7), zero)
        o["e"], o["p"] = e, p
        o["v"] = torch.where((vnew - 1.0).abs() < 1e-10, torch.ones_like(vnew), vnew)
        # the next time step's limits
        moving = vdov != 0.0
        far = torch.full_like(vdov, math.inf)
        c = o["ss"] ** 2 + torch.where(vdov < 0.0, 256.0 * arealg ** 2 * vdov ** 2, zero)
        courant = torch.where(moving, arealg / c.sqrt(), far)
        hydro = torch.where(moving, 0.1 / (vdov.abs() + 1e-20), far)
        for name, lim in (("dtcourant", courant), ("dthydro", hydro)):
            least = lim[torch.argmin(lim)]
            o[name] = least if float(least) < 1e20 else s[name]
        return o


    def run(self, s, cycles, keep=False):
        """Up to `cycles` cycles to the stop time: the states (with `keep`, all of them)."""
        states = [s]
        with torch.no_grad():
            while states[-1]["cycle"] < cycles and float(states[-1]["time"]) < 1e-2:
                states = (states if keep else []) + [self.step(states[-1])]
        return states


def _tensors(fields, scalars, device):
    s = {k: torch.from_numpy(np.ascontiguousarray(f)).to(device) for k, f in fields.items()}
    s |= {k: torch.tensor(float(v), dtype=torch.float64, device=device) for k, v in scalars.items() if k != "cycle"}
    s["cycle"] = scalars["cycle"]
    return s


def _exact_ensemble(case, seed):
    out = {"e": [], "x": [], "time": []}
    for spec in _instances(case, seed):
        nx = spec["nx"]
        m = _Sedov(nx, case["mode"], _device())
        zero = torch.zeros_like(m.volo)
        e = zero.clone()
        e[0] = spec["einit"]
        s = dict(zip(STATE, (*m.X, *torch.zeros_like(m.X), e, zero, zero, zero + 1, zero)))
        dt = 0.5 * float(m.volo[0]) ** (1 / 3) / math.sqrt(2.0 * spec["einit"])
        s |= {k: torch.tensor(v, dtype=torch.float64, device=m.device)
              for k, v in (("time", 0.0), ("deltatime", dt), ("dtcourant", 1e20), ("dthydro", 1e20), ("hgcoef", spec["hgcoef"]))}
        s["cycle"] = 0
        s = m.run(s, case["cycles"])[-1]
        out["e"].append(s["e"].cpu().numpy())
        out["x"].append(s["x"].cpu().numpy())
        out["time"].append(np.array([float(s["time"])]))
    return {k: np.concatenate(v) for k, v in out.items()}


def _exact_adjoint(case, m, s):
    """The objective's value and gradient, one cycle's graph at a time."""
    carried = STATE + ("time", "deltatime", "dtcourant", "dthydro")
    states = m.run(s, case["cycles"], keep=True)
    h, r2 = EDGE / m.nx, 0.3 ** 2
    we = torch.where((m.X[:, m.nl[0]] + 0.5 * h).square().sum(0) < r2, m.volo, torch.zeros_like(m.volo))
    wn = torch.where(m.X.square().sum(0) < r2, m.mass, torch.zeros_like(m.mass))
    end = states[-1]
    loss = (we * end["e"]).sum() + 0.5 * (wn * (end["xd"] ** 2 + end["yd"] ** 2 + end["zd"] ** 2)).sum()
    bar = {k: torch.zeros_like(end[k]) for k in carried}
    bar["e"] = we.clone()
    for k in ("xd", "yd", "zd"):
        bar[k] = wn * end[k]
    hg = 0.0
    for before in reversed(states[:-1]):
        names = carried + ("hgcoef",)
        leaf = {k: before[k].detach().clone().requires_grad_(True) for k in names}
        after = m.step({**before, **leaf})
        pairs = [(after[k], bar[k]) for k in carried if after[k].requires_grad]
        got = torch.autograd.grad([a for a, _ in pairs], [leaf[k] for k in names], [b for _, b in pairs], allow_unused=True)
        got = {k: torch.zeros_like(leaf[k]) if g is None else g for k, g in zip(names, got)}
        hg += float(got["hgcoef"])
        bar = {k: got[k] for k in carried}
    return {"loss": float(loss), "hgcoef": hg, **{k: bar[k].cpu().numpy() for k in STATE}}


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        return _exact_ensemble(case, seed) if case["n"] * case["cycles"] <= 2000 else None
    nx, tp = case["nx"], case.get("blocks", 1)
    m = _Sedov(nx * tp, case["mode"], _device())
    s = _tensors(*_blast(nx * tp, seed), m.device)
    if kind == "adjoint":
        return _exact_adjoint(case, m, s)
    with torch.no_grad():
        if kind == "force":
            f = m.forces(s)
            return {"fx": f[0], "fy": f[1], "fz": f[2]}
        s = m.run(s, case["cycles"])[-1]
    out = {k: s[k].cpu().numpy() for k in STATE}
    if tp > 1:
        eg, ng = _block_ids(nx, tp)
        out = {k: f[ng if k in NODE else eg] for k, f in out.items()}
    out["time"] = float(s["time"])
    return out
