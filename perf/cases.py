"""The framework's work as its users have it done, for timing and for comparing outputs:
ring impacts (updated and total Lagrangian), the pulled plate (weak form), batched
ensembles, the surrogate's data generation, and the surrogate itself.

``listed()`` names the cases, ``draw()`` gives more of the same ranges, ``prepare()``
makes the inputs from a seed and the objects a program keeps, ``run()`` is one pass,
``work()`` what a pass cannot do without, and ``exact()`` the same outputs in plain
64-bit torch (no library code beyond the scenario builders that lay out the inputs).

A pass of a simulation sets the initial state (pinned host arrays), advances it and reads
the state back, the loop of a program that runs one initial state after another; the weak
form, whose Gauss-point state the library keeps, goes on from where it is.  Velocities,
densities and stresses of the mixed form are handed on in 32 bits, the precision of its
pair sums; positions, and every field of the 64-bit forms, in 64.
"""
import ctypes
import math

import numpy as np
import torch

import mfree_iwf_gb300 as M
from mfree_iwf_gb300 import scenarios as S
from mfree_iwf_gb300 import surrogate as G

FIELDS = ("x", "y", "vx", "vy", "rho", "Sxx", "Sxy", "Syy")
R_OUT, BATCH, DIMS = 0.04, 512, (6, 256, 256, 256, 66)


def listed():
    return [
        # the integration guide's loop: one body, the default parity form, a step a call
        {"name": "rings_ul_strict_1mm", "kind": "ul", "form": "fp64_strict", "nbox": 81, "calls": 10, "steps": 1,
         "graph": False, "tune": False},
        # the same rings in the production form, replayed from a captured step
        {"name": "rings_ul_mixed_1mm", "kind": "ul", "form": "mixed", "nbox": 81, "calls": 1, "steps": 100,
         "graph": True, "tune": False},
        # the headline benchmark: 1.76M particles with contact, autotuned as the benchmark does
        {"name": "rings_tl_mixed_50um", "kind": "tl", "form": "mixed", "nbox": 1601, "calls": 1, "steps": 20,
         "graph": True, "tune": True},
        # the plain 64-bit form the benchmark compares it with, a quarter of the particles
        {"name": "rings_tl_fp64_100um", "kind": "tl", "form": "fp64", "nbox": 801, "calls": 1, "steps": 5,
         "graph": True, "tune": True},
        # plate tension, weak form with RKPM: 0.8M particles, 3.2M Gauss points
        {"name": "plate_weak_mixed_50um", "kind": "plate", "form": "mixed", "nbox": 2001, "calls": 1, "steps": 20,
         "graph": True, "tune": False},
        # the same in 64 bits at a parity study's size
        {"name": "plate_weak_fp64_200um", "kind": "plate", "form": "fp64", "nbox": 501, "calls": 1, "steps": 5,
         "graph": True, "tune": False},
        # batched ensemble of uneven ring impacts (4k to 110k particles each), autotuned
        {"name": "ensemble_mixed_64", "kind": "ensemble", "form": "mixed", "nbox": 64, "calls": 1, "steps": 20,
         "graph": True, "tune": True},
        # its plain 64-bit form
        {"name": "ensemble_fp64_16", "kind": "ensemble", "form": "fp64", "nbox": 16, "calls": 1, "steps": 3,
         "graph": True, "tune": True},
        # the surrogate's data generation: many small two-body impacts, contact, monitor
        {"name": "sweep_mixed_256", "kind": "sweep", "form": "mixed", "nbox": 256, "calls": 1, "steps": 10,
         "graph": True, "tune": False},
        # a screened sweep's network pass: 10,000 rows from and to host arrays
        {"name": "surrogate_screen_10k", "kind": "predict", "rows": 10000, "host": True},
        # the network alone over device-resident rows
        {"name": "surrogate_predict_262k", "kind": "predict", "rows": 262140, "host": False},
        # training steps of the five-member ensemble
        {"name": "surrogate_train_50", "kind": "train", "rows": 4000, "steps": 50},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ul", "tl", "tl", "plate", "ensemble", "sweep", "predict", "train"])
    if kind == "predict":
        return {"kind": kind, "rows": _log_int(rng, 1, 262140), "host": rng.random() < 0.5}
    if kind == "train":
        return {"kind": kind, "rows": _log_int(rng, 500, 20000), "steps": rng.randint(5, 50)}
    form = rng.choice(["mixed", "mixed", "fp64", "fp64_strict"])
    wide = form == "mixed"
    nbox = {"ul": _log_int(rng, 61, 801 if wide else 161), "tl": _log_int(rng, 61, 1601 if wide else 401),
            "plate": _log_int(rng, 101, 1501 if wide else 401), "ensemble": _log_int(rng, 2, 48 if wide else 6),
            "sweep": _log_int(rng, 4, 256 if wide else 32)}[kind]
    return {"kind": kind, "form": form, "nbox": nbox, "calls": 1,
            "steps": rng.randint(2, 10) if wide else rng.randint(1, 3), "graph": rng.random() < 0.7, "tune": False}


# ------------------------------------------------------------------ inputs
def _scenario(case, seed):
    """The scenario (constants, bodies, boundary conditions) and contact groups."""
    k, n = case["kind"], case["nbox"]
    if k == "ul":
        return S.c1_rings(dx=2 * R_OUT / (n - 1)), None
    if k == "tl":
        return S.c2_rings_tl(dx=2 * R_OUT / (n - 1)), None
    if k == "plate":
        return S.c3_plate(dx=0.1 / (n - 1), seed=seed), None
    if k == "ensemble":
        return S.c4_ensemble(n), None
    return G.batch_scenario(G.sample_params(n, 11))


def _columns(sc):
    """The bodies' rows one after another, and per row its body."""
    col = {f: np.concatenate([b.arrays[f] for b in sc.bodies]) for f in FIELDS + ("X", "Y", "m", "h")}
    col["body"] = np.repeat(np.arange(len(sc.bodies)), [b.n for b in sc.bodies])
    return col


def _body_values(sc, key):
    return np.array([(b.params or {}).get(key, getattr(sc, key)) for b in sc.bodies], np.float64)


def _state(case, sc, seed):
    """A deformed, vibrating state on the scenario's lattice: strains of some 1e-3 and, in
    the updated-Lagrangian forms, densities and stresses of that size, from the seed."""
    c = _columns(sc)
    rng = np.random.default_rng(seed)

    def wave(size):
        """a sum of three plane waves over the body, amplitude about `size`"""
        out = 0.0
        for _ in range(3):
            kx, ky = rng.uniform(-2, 2, 2) * 2 * np.pi / R_OUT
            out = out + np.sin(kx * c["x"] + ky * c["y"] + rng.uniform(0, 6.28))
        return size / 3 * out

    E = _body_values(sc, "E")[c["body"]]
    new = {f: c[f].copy() for f in FIELDS}
    speed = np.abs(c["vx"]) + (1.0 if case["kind"] == "plate" else 0.0)
    new["vx"] += 0.02 * speed * wave(1.0)
    new["vy"] += 0.02 * speed * wave(1.0)
    if case["kind"] == "plate":
        new["vx"] += 20.0 * (c["x"] - 0.05)  # the stretch that the pulled ends impose
        return new
    if case["kind"] == "tl":
        new["x"] += wave(1e-5)
        new["y"] += wave(1e-5)
        return new
    new["rho"] *= 1.0 + wave(1e-3)
    for f in ("Sxx", "Sxy", "Syy"):
        new[f] += E * wave(1e-3)
    return new


def _pinned(n):
    return torch.empty(n, dtype=torch.float64).pin_memory()


class Run:
    """What a program keeps: the simulation, its pinned state arrays, 32-bit copies."""

    def __init__(self, case, seed):
        sc, groups = _scenario(case, seed)
        self.case, self.n = case, sc.n_total
        state = _state(case, sc, seed)
        self.reset = case["kind"] != "plate"
        if not self.reset:  # the weak form starts from the scenario's own arrays
            for f in FIELDS:
                sc.bodies[0].arrays[f] = state[f]
        self.sim = M.from_scenario(sc, precision=case["form"], groups=groups, graph=case["graph"])
        self.sim.step(0)  # set-up: neighbour lists and corrections
        self.host_in = {f: _pinned(self.n) for f in FIELDS}
        for f in FIELDS:
            self.host_in[f].copy_(torch.from_numpy(state[f]))
        self.into = {f: t.numpy() for f, t in self.host_in.items()}
        self.host_out = {f: _pinned(self.n) for f in FIELDS}
        self.out = {f: t.numpy() for f, t in self.host_out.items()}
        self.narrow = {f: torch.empty(self.n, dtype=torch.float32) for f in FIELDS[2:]} if case["form"] == "mixed" else {}
        if case["tune"]:
            self.sim.autotune(1)
        if case["kind"] == "sweep":
            self.sim.set_monitor(case["steps"])
        if self.reset:
            self.sim.set_state_all(self.into)
            self.sim.step(case["steps"])  # captures the step

    def run(self):
        if self.reset:
            self.sim.set_state_all(self.into)
        for _ in range(self.case["calls"]):
            self.sim.step(self.case["steps"])
        self.sim.get_state_all_into(self.out)
        got = dict(self.host_out)
        for f, t in self.narrow.items():
            got[f] = t.copy_(self.host_out[f])
        if self.case["kind"] == "sweep":
            got["monitor"] = self.sim.monitor()
        return got


def _weights(seed, members=5):
    """[members][parameters], per layer W [out][in] (He-uniform) then b, as the model takes them."""
    rng = np.random.default_rng(seed)
    rows = []
    for _ in range(members):
        parts = []
        for i, o in zip(DIMS[:-1], DIMS[1:]):
            parts += [rng.uniform(-1, 1, i * o) * math.sqrt(6.0 / i), rng.uniform(-0.1, 0.1, o)]
        rows.append(np.concatenate(parts))
    return np.stack(rows).astype(np.float32)


def _rows(n, seed):
    return np.random.default_rng(seed + 1).uniform(-1, 1, (n, DIMS[0])).astype(np.float32)


def _targets(x, seed):
    """Smooth z-scored targets of the surrogate's kind."""
    w = np.random.default_rng(seed + 2).normal(size=(DIMS[0], DIMS[-1]))
    return np.sin(x.astype(np.float64) @ w).astype(np.float32)


class Net:
    def __init__(self, case, seed):
        self.case = case
        self.mlp = G.Mlp(DIMS, members=5, max_batch=BATCH, seed=seed % (1 << 31))
        for z, p in enumerate(_weights(seed)):
            self.mlp.set_params(z, p)
        self.x = _rows(case["rows"], seed)
        if case["kind"] == "train":
            self.mlp.set_data(self.x, _targets(self.x, seed))
        elif not case["host"]:
            self.x = torch.from_numpy(self.x).cuda()
            self.y = torch.empty(5, case["rows"], DIMS[-1], device="cuda")

    def run(self):
        mlp = self.mlp
        if self.case["kind"] == "train":
            hist = mlp.train(self.case["steps"], 2e-3, 2e-5)
            return {"loss": hist, "params": [mlp.get_params(z) for z in range(5)]}
        if self.case["host"]:
            return mlp.predict(self.x)
        fp = ctypes.POINTER(ctypes.c_float)
        mlp._check(mlp._lib.mf_mlp_predict(mlp._h, ctypes.cast(self.x.data_ptr(), fp), len(self.x),
                                           ctypes.cast(self.y.data_ptr(), fp)), "mf_mlp_predict")
        return self.y


def prepare(case, seed):
    return (Net if case["kind"] in ("predict", "train") else Run)(case, seed)


def run(state):
    return state.run()


# -------------------------------------------------------------------- work
def work(case):
    """Per step and particle: the state read and written once, and per stage and pair the
    arithmetic of the pair terms; per row and member: inputs, outputs and the products."""
    if case["kind"] in ("predict", "train"):
        macs = sum(a * b for a, b in zip(DIMS[:-1], DIMS[1:]))
        if case["kind"] == "train":
            params = 5 * (macs + sum(DIMS[1:]))
            return {"bytes": case["steps"] * params * 24.0, "flops": case["steps"] * 6.0 * macs * BATCH * 5}
        return {"bytes": 4.0 * case["rows"] * (DIMS[0] + 5 * DIMS[-1]), "flops": 10.0 * macs * case["rows"]}
    k, nbox, steps = case["kind"], case["nbox"], case["calls"] * case["steps"]
    ring = math.pi * (1 - 0.75 ** 2) / 4
    n = {"ul": 2 * ring * nbox ** 2, "tl": 2 * ring * nbox ** 2, "plate": nbox * (0.2 * nbox + 1),
         "ensemble": 21000.0 * nbox, "sweep": 1240.0 * nbox}[k]
    mixed = case["form"] == "mixed"
    state = {"tl": 32, "plate": 32 + 4 * (16 if mixed else 32)}.get(k, 48 if mixed else 64)
    flops = {"tl": 21 * 60.0, "plate": 4 * 21 * 24.0}.get(k, 21 * 110.0)
    return {"bytes": n * (steps * 2.0 * state + (2.0 if k != "plate" else 1.0) * 64), "flops": n * steps * 4 * flops}


# ------------------------------------------------------------------- exact
def _gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _pairs(px, py, pbody, qx, qy, qbody, radius):
    """(i, j): the points j of q within `radius` (per body) of each point i of p."""
    nb = len(radius)
    lo = [torch.full((nb,), 1e300, device="cuda", dtype=torch.float64).scatter_reduce(0, qbody, a, "amin") for a in (qx, qy)]
    cell = lambda a, body, l: torch.floor((a - l[body]) / radius[body]).long() + 1  # noqa: E731
    cx, cy = cell(qx, qbody, lo[0]), cell(qy, qbody, lo[1])
    size = [torch.zeros(nb, device="cuda", dtype=torch.long).scatter_reduce(0, qbody, a, "amax") + 3 for a in (cx, cy)]
    off = torch.cumsum(size[0] * size[1], 0) - size[0] * size[1]
    key, order = torch.sort(off[qbody] + cx * size[1][qbody] + cy)
    start = torch.searchsorted(key, torch.arange(int((size[0] * size[1]).sum()) + 1, device="cuda"))
    home = off[pbody] + cell(px, pbody, lo[0]).clamp(1, None).minimum(size[0][pbody] - 2) * size[1][pbody] \
        + cell(py, pbody, lo[1]).clamp(1, None).minimum(size[1][pbody] - 2)
    found = []
    for d in (-1, 0, 1):
        row = home + d * size[1][pbody]
        s, e = start[row - 1], start[row + 2]
        i = torch.repeat_interleave(torch.arange(len(px), device="cuda"), e - s)
        j = order[torch.arange(len(i), device="cuda") - (torch.cumsum(e - s, 0) - (e - s) - s)[i]]
        near = (px[i] - qx[j]) ** 2 + (py[i] - qy[j]) ** 2 <= radius[pbody][i] ** 2
        found.append((i[near], j[near]))
    return torch.cat([f[0] for f in found]), torch.cat([f[1] for f in found])


def _spline(dx, dy, h):
    """The cubic spline W and its gradient at the offset (dx, dy)."""
    r = torch.sqrt(dx * dx + dy * dy)
    q, fac = r / h, 10 / (7 * math.pi) / h ** 2
    t = (2 - q).clamp(min=0)
    w = torch.where(q < 1, 1 - 1.5 * q * q * (1 - 0.5 * q), 0.25 * t ** 3) * fac
    d = torch.where(q < 1, -3 * q * (1 - 0.75 * q), -0.75 * t * t) * fac / h / r.clamp(min=1e-300)
    return w, dx * d, dy * d


def _sum(i, n, v):
    return torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, i, v)


def _viscosity(k, i, j, x, y, vx, vy, rho, h, c, mass_grad):
    """Monaghan's artificial viscosity as accelerations."""
    dx, dy, dvx, dvy = x[i] - x[j], y[i] - y[j], vx[i] - vx[j], vy[i] - vy[j]
    dot = (dvx * dx + dvy * dy).clamp(max=0)
    hij, rij, cij = 0.5 * (h[i] + h[j]), 0.5 * (rho[i] + rho[j]), 0.5 * (c[i] + c[j])
    mu = hij * dot / (dx * dx + dy * dy + k["eta"] ** 2 * hij * hij)
    pi = (-k["alpha"] * cij * mu + k["beta"] * mu * mu) / rij
    return [_sum(i, len(x), -pi * g) for g in mass_grad]


def _jaumann(l, s, shear):
    xx, xy, yx, yy = l
    tr = (xx + yy) / 3
    w = 0.5 * (xy - yx)
    return (2 * shear * (xx - tr) + 2 * w * s[1], shear * (xy + yx) + w * (s[2] - s[0]), 2 * shear * (yy - tr) - 2 * w * s[1])


def _rk4(state, dt, rates, begin=None):
    """One classical step of a list of arrays."""
    total, now = None, state
    for stage, (c, w) in enumerate(((0.5, 1), (0.5, 2), (1.0, 2), (0, 1))):
        if begin:
            now = begin(now)
        k = rates(now)
        total = k if stage == 0 else [a + w * b for a, b in zip(total, k)]
        if stage < 3:
            now = [a + c * dt * b for a, b in zip(state, k)]
    return [a + dt / 6 * b for a, b in zip(state, total)]


def _ul(case, sc, start):
    col = _columns(sc)
    body, m, h = (_gpu(col[f]) for f in ("body", "m", "h"))
    per = lambda key: _gpu(_body_values(sc, key))[body]  # noqa: E731
    E, nu, rho0, dt, wdx = (per(key) for key in ("E", "nu", "rho0", "dt", "wdeltap"))
    K, shear = E / (3 * (1 - 2 * nu)), E / (2 * (1 + nu))
    s = [_gpu(start[f]) for f in FIELDS]
    n, hb = len(m), torch.zeros(len(sc.bodies), dtype=torch.float64, device="cuda").scatter_(0, body, h)
    i, j = _pairs(s[0], s[1], body, s[0], s[1], body, 2.2 * hb)
    i, j = i[i != j], j[i != j]
    const = {"alpha": sc.alpha, "beta": sc.beta, "eta": sc.eta}

    def rates(st):
        x, y, vx, vy, rho, sxx, sxy, syy = st
        p = K / rho0 * (rho - rho0)
        a, b = sxx - p, syy - p
        th = 0.5 * torch.atan2(2 * sxy, a - b)
        cs, sn = torch.cos(th), torch.sin(th)
        ra = -sc.mghn_eps * (cs * cs * a + 2 * cs * sn * sxy + sn * sn * b).clamp(min=0) / rho ** 2
        rb = -sc.mghn_eps * (sn * sn * a - 2 * cs * sn * sxy + cs * cs * b).clamp(min=0) / rho ** 2
        rxx, rxy, ryy = cs * cs * ra + sn * sn * rb, cs * sn * (ra - rb), sn * sn * ra + cs * cs * rb
        w, gx, gy = _spline(x[i] - x[j], y[i] - y[j], h[i])
        f = (w / wdx[i]) ** sc.corr_exp
        pair = lambda v, r: m[j] * ((v / rho ** 2)[i] + (v / rho ** 2)[j] + f * (r[i] + r[j]))  # noqa: E731
        txy = pair(sxy, rxy)
        fx = _sum(i, n, pair(a, rxx) * gx + txy * gy)  # rho and 1 / rho of the momentum cancel
        fy = _sum(i, n, txy * gx + pair(b, ryy) * gy)
        dvx, dvy, q = vx[j] - vx[i], vy[j] - vy[i], (m / rho)[j]
        l = [_sum(i, n, d * g * q) for d in (dvx, dvy) for g in (gx, gy)]
        av = _viscosity(const, i, j, x, y, vx, vy, rho, h, torch.sqrt(K / rho), (m[j] * gx, m[j] * gy))
        xs = sc.xsph_eps * w * m[i] / (0.5 * (rho[i] + rho[j]))
        ds = _jaumann(l, (sxx, sxy, syy), shear)
        return [vx + _sum(i, n, xs * dvx), vy + _sum(i, n, xs * dvy), fx + av[0], fy + av[1], -rho * (l[0] + l[3]), *ds]

    rows = []
    for _ in range(case["calls"] * case["steps"]):
        s = _rk4(s, dt, rates)
        if case["kind"] == "sweep":  # the monitor's row; the rings do not touch yet
            p = K / rho0 * (s[4] - rho0)
            a, b = s[5] - p, s[7] - p
            vm = torch.sqrt(a * a - a * b + b * b + 3 * s[6] ** 2)
            nb = len(sc.bodies)
            cnt = _sum(body, nb, torch.ones_like(m))
            top = torch.zeros(nb, dtype=torch.float64, device="cuda").scatter_reduce(0, body, vm, "amax")
            rows.append(torch.stack([_sum(body, nb, s[2]) / cnt, _sum(body, nb, s[3]) / cnt, top, 0 * top], 1))
    out = dict(zip(FIELDS, s))
    if rows:
        out["monitor"] = torch.stack(rows)
    return out


def _nominal(hxx, hxy, hyx, hyy, sxx, sxy, syy):
    """J F^-1 sigma."""
    a, b, c, d = 1 + hyy, -hxy, -hyx, 1 + hxx
    return a * sxx + b * sxy, a * sxy + b * syy, c * sxx + d * sxy, c * sxy + d * syy


def _tl(case, sc, start):
    col = _columns(sc)
    body, m, h, X, Y = (_gpu(col[f]) for f in ("body", "m", "h", "X", "Y"))
    n, rho0, K = len(m), sc.rho0, sc.E / (3 * (1 - 2 * sc.nu))
    hb = torch.zeros(len(sc.bodies), dtype=torch.float64, device="cuda").scatter_(0, body, h)
    i, j = _pairs(X, Y, body, X, Y, body, 2.0 * hb)
    w, gx, gy = _spline(X[i] - X[j], Y[i] - Y[j], h[i])
    v = m / rho0
    C = _sum(i, n, w * v[j])
    dx, dy = X[j] - X[i], Y[j] - Y[i]
    b00, b10, b01, b11 = (_sum(i, n, d * g * v[j]) / C for d, g in ((dx, gx), (dx, gy), (dy, gx), (dy, gy)))
    det = (b00 * b11 - b10 * b01) * C
    gx, gy = gx * (b11 / det)[i] - gy * (b10 / det)[i], gy * (b00 / det)[i] - gx * (b01 / det)[i]
    const = {"alpha": sc.alpha, "beta": sc.beta, "eta": sc.eta}
    s = [_gpu(start[f]) for f in FIELDS]
    keep = s[4:]
    c = torch.sqrt(K / keep[0])
    D = sc.E / (1 - sc.nu ** 2)

    def rates(st):
        x, y, vx, vy = st
        ux, uy = x - X, y - Y
        hxx, hxy, hyx, hyy = (_sum(i, n, (u[j] - u[i]) * g * v[j]) for u in (ux, uy) for g in (gx, gy))
        e00, e11 = hxx + 0.5 * (hxx * hxx + hyx * hyx), hyy + 0.5 * (hxy * hxy + hyy * hyy)
        e01 = 0.5 * (hxy + hyx + hxx * hxy + hyx * hyy)
        pxx, pxy, pyx, pyy = _nominal(hxx, hxy, hyx, hyy, D * (e00 + sc.nu * e11), D * (1 - sc.nu) * e01, D * (sc.nu * e00 + e11))
        mg = (m[j] * gx, m[j] * gy)
        ax = _sum(i, n, (pxx[i] + pxx[j]) * mg[0] + (pyx[i] + pyx[j]) * mg[1]) / rho0 ** 2
        ay = _sum(i, n, (pxy[i] + pxy[j]) * mg[0] + (pyy[i] + pyy[j]) * mg[1]) / rho0 ** 2
        av = _viscosity(const, i, j, x, y, vx, vy, keep[0], h, c, mg)
        return [vx, vy, ax + av[0], ay + av[1]]

    s = s[:4]
    for _ in range(case["calls"] * case["steps"]):
        s = _rk4(s, sc.dt, rates)
    return dict(zip(FIELDS, s + keep))


def _rkpm(px, py, i, j, X, Y, h, v):
    """RKPM functions and gradients (linear basis) of the points p over the pairs (i, j)."""
    n = len(px)
    rx, ry = (px[i] - X[j]) / h, (py[i] - Y[j]) / h
    w, gx, gy = _spline(rx, ry, 1.0)
    one, o = torch.ones_like(rx), torch.zeros_like(rx)
    base, slope = (one, rx, ry), ((o, one, o), (o, o, one))

    def moments(f):
        m = torch.zeros(n, 3, 3, dtype=torch.float64, device="cuda")
        for a in range(3):
            for b in range(a + 1):
                m[:, a, b] = m[:, b, a] = _sum(i, n, f(a, b) * v[j])
        return m

    A = moments(lambda a, b: w * base[a] * base[b])
    inv = torch.linalg.inv(A)
    C = inv[:, :, 0]
    corr = sum(C[i, a] * base[a] for a in range(3))
    out = [w * corr]
    for g, d in ((gx, slope[0]), (gy, slope[1])):
        B = moments(lambda a, b: g * base[a] * base[b] + w * (d[a] * base[b] + base[a] * d[b]))
        Cd = -(inv @ (B @ C[:, :, None]))[:, :, 0]
        cd = sum(Cd[i, a] * base[a] + C[i, a] * d[a] for a in range(3))
        out.append((g * corr + w * cd) / h)
    return out


def _plate(case, sc, start):
    b = sc.bodies[0]
    X, Y, m = (_gpu(b.arrays[f]) for f in ("X", "Y", "m"))
    n, rho0, h = len(m), sc.rho0, sc.nbh_h
    v = m / rho0
    nodes = torch.arange(n, device="cuda").reshape(b.ey + 1, b.ex + 1)
    ll, lr, tr, tl = (t.reshape(-1) for t in (nodes[:-1, :-1], nodes[:-1, 1:], nodes[1:, 1:], nodes[1:, :-1]))
    gx, gy, gw = [], [], []
    p = 0.577350269189626
    for xi in (p, -p):
        for eta in (p, -p):
            N = [0.25 * (1 + a * xi) * (1 + c * eta) for a, c in ((-1, -1), (1, -1), (1, 1), (-1, 1))]
            Nx = [0.25 * a * (1 + c * eta) for a, c in ((-1, -1), (1, -1), (1, 1), (-1, 1))]
            Ne = [0.25 * c * (1 + a * xi) for a, c in ((-1, -1), (1, -1), (1, 1), (-1, 1))]
            at = lambda q, f: sum(k * q[e] for k, e in zip(f, (ll, lr, tr, tl)))  # noqa: E731
            gx.append(at(X, N))
            gy.append(at(Y, N))
            gw.append(-(at(X, Nx) * at(Y, Ne) - at(X, Ne) * at(Y, Nx)))
    gx, gy, gw = (torch.stack(t, 1).reshape(-1) for t in (gx, gy, gw))
    ng = len(gx)
    one = lambda k: torch.zeros(k, dtype=torch.long, device="cuda")  # noqa: E731
    r = torch.tensor([2.0 * h], dtype=torch.float64, device="cuda")
    i, j = _pairs(gx, gy, one(ng), X, Y, one(n), r)
    _, wx, wy = _rkpm(gx, gy, i, j, X, Y, h, v / h ** 2)
    wx, wy = wx / h ** 2, wy / h ** 2
    pi, pj = _pairs(X, Y, one(n), X, Y, one(n), r)
    pw = _rkpm(X, Y, pi, pj, X, Y, h, v / h ** 2)[0] / h ** 2 * v[pj]
    K, shear = sc.E / (3 * (1 - 2 * sc.nu)), sc.E / (2 * (1 + sc.nu))
    qx, qy = wx * v[j], wy * v[j]
    s = [_gpu(start[f]) for f in FIELDS[:4]]
    g = [torch.full((ng,), sc.gp_rho, dtype=torch.float64, device="cuda")] + [torch.zeros(ng, dtype=torch.float64, device="cuda") for _ in range(3)]
    t = 0.0

    def pull(st, time):
        st = [a.clone() for a in st]
        for bc in b.bcs:
            k = _gpu(bc.idx.astype(np.int64))
            st[0][k], st[1][k], st[2][k], st[3][k] = X[k] + bc.v * time, Y[k], bc.v, 0.0
        return st

    def rates(st):
        x, y, vx, vy, rho, sxx, sxy, syy = st
        hxx, hxy, hyx, hyy = (_sum(i, ng, u[j] * q) for u in (x - X, y - Y) for q in (qx, qy))
        fxx, fxy, fyx, fyy = (_sum(i, ng, u[j] * q) for u in (vx, vy) for q in (qx, qy))
        J = (1 + hxx) * (1 + hyy) - hxy * hyx
        l = ((fxx * (1 + hyy) - fxy * hyx) / J, (fxy * (1 + hxx) - fxx * hxy) / J,
             (fyx * (1 + hyy) - fyy * hyx) / J, (fyy * (1 + hxx) - fyx * hxy) / J)
        pr = K / rho0 * (rho - rho0)
        pxx, pxy, pyx, pyy = _nominal(hxx, hxy, hyx, hyy, sxx - pr, sxy, syy - pr)
        ax = -_sum(j, n, ((pxx * gw)[i] * qx + (pyx * gw)[i] * qy)) / m
        ay = -_sum(j, n, ((pxy * gw)[i] * qx + (pyy * gw)[i] * qy)) / m
        return [vx, vy, ax, ay, -rho * (l[0] + l[3]), *_jaumann(l, (sxx, sxy, syy), shear)]

    for _ in range(case["calls"] * case["steps"]):
        full = _rk4(s + g, sc.dt, rates, lambda st: pull(st[:4], t) + st[4:])
        t += sc.dt
        s, g = pull(full[:4], t), full[4:]
        if sc.do_smooth:
            s[2], s[3] = (_sum(pi, n, a[pj] * pw) for a in s[2:4])
    return dict(zip(FIELDS, s + [_gpu(start[f]) for f in FIELDS[4:]]))


def _layers(flat):
    """The members' parameters as per-layer (W [members][out][in], b [members][out])."""
    o, out = 0, []
    for i, k in zip(DIMS[:-1], DIMS[1:]):
        out.append([flat[:, o:o + i * k].reshape(-1, k, i), flat[:, o + i * k:o + i * k + k]])
        o += i * k + k
    return out


def _forward(layers, x):
    acts = [x]
    for k, (w, b) in enumerate(layers):
        z = acts[-1] @ w.transpose(1, 2) + b[:, None, :]
        acts.append(z.clamp(min=0) if k + 1 < len(layers) else z)
    return acts


def _splitmix(x):
    with np.errstate(over="ignore"):
        x = x + np.uint64(0x9E3779B97F4A7C15)
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return x ^ (x >> np.uint64(31))


def _train(case, seed):
    """Adam on bootstrap minibatches, the draws those of the model's seeded hash."""
    x = _rows(case["rows"], seed)
    xd, yd = _gpu(x.astype(np.float64)), _gpu(_targets(x, seed).astype(np.float64))
    p = _gpu(_weights(seed).astype(np.float64))
    m, v, losses, steps = torch.zeros_like(p), torch.zeros_like(p), [], case["steps"]
    key = np.uint64(((seed % (1 << 31)) * 0x2545F4914F6CDD1D + 1) % (1 << 64))
    z, r = np.arange(5, dtype=np.uint64)[:, None] << np.uint64(52), np.arange(BATCH, dtype=np.uint64)
    for t in range(1, steps + 1):
        src = _gpu((_splitmix(key ^ np.uint64(t << 20) ^ z ^ r) % np.uint64(case["rows"])).astype(np.int64))
        layers = _layers(p)
        acts = _forward(layers, xd[src])
        d = acts[-1] - yd[src]
        losses.append((d * d).mean((1, 2)))
        d, parts = d * (2 / (BATCH * DIMS[-1])), []
        for k in reversed(range(len(layers))):
            parts = [(d.transpose(1, 2) @ acts[k]).reshape(5, -1), d.sum(1)] + parts
            d = d @ layers[k][0] * (acts[k] > 0)
        grad = torch.cat(parts, 1)
        frac = (t - 1) / (steps - 1) if steps > 1 else 0.0
        lr = 2e-5 + 0.5 * (2e-3 - 2e-5) * (1 + math.cos(math.pi * frac))
        m, v = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad * grad
        p = p - lr * (m / (1 - 0.9 ** t)) / (torch.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
    return {"loss": torch.stack(losses), "params": list(p)}


def exact(case, seed):
    if case["kind"] == "train":
        return _train(case, seed)
    if case["kind"] == "predict":
        layers = _layers(_gpu(_weights(seed).astype(np.float64)))
        out = torch.empty(5, case["rows"], DIMS[-1], dtype=torch.float64, device="cuda")
        x = _gpu(_rows(case["rows"], seed).astype(np.float64))
        for r in range(0, len(x), 32768):
            out[:, r:r + 32768] = _forward(layers, x[r:r + 32768].expand(5, -1, -1))[-1]
        return out
    sc, _ = _scenario(case, seed)
    start = _state(case, sc, seed)
    with torch.no_grad():
        return {"tl": _tl, "plate": _plate}.get(case["kind"], _ul)(case, sc, start)
