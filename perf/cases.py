"""Timed cases of the MPH-I engine: what its users have it do, through `mphimplicit_gb300.engine`.

A case is one request on a simulation state in host memory.  Its `entry`:

  advance  the state goes up (`Case.set_state`), `steps` time steps are taken (`Case.step`), the new state comes
           back (`Case.fields`): a time loop that keeps its case and exchanges states, as a coupled program does
  frame    the same with the fields of an output frame (`stage("output_fields")`, every field of `Case.fields`)
  batch    `advance` for `count` independent 2D cases at once (`engine.batch_step`)
  job      a case created from the particles, stepped, read and closed: a request of a server, a short run

The geometries and constants are those of `casegen`: a block of fluid in the lower corner of a closed box of wall
particles (2D: l0 = 0.01 m, dt = 1e-4 s; 3D: l0 = 0.005 m, dt = 5e-5 s).  The fluid turns over slowly (a vortex of
a few tenths of the free-fall speed with a little noise), as it does in the middle of a run; the particles are
jittered by 1 % of their spacing.  `form` is the solver form: "mixed" (refined to `tol`, the start value
extrapolated from the steps before) or "fp64" (the reference's algorithm with its own stop test).

`exact` is the time step of the method in plain torch, 64 bits throughout and without this repository's kernels,
its linear system solved to rounding.
"""
import dataclasses
import math

import numpy as np
import torch

from mphimplicit_gb300 import casegen, engine
from mphimplicit_gb300.cabi import PRECISION_FP64, PRECISION_MIXED

EXACT_MAX = 420_000   # particles (times steps / 2) up to which `exact` stays within some twenty seconds


def _case(entry, dim, form, fluid, steps, mu=0.1, two=False, tension=0.0, lid=False, count=1, tol=1e-10):
    fx, fy, fz = tuple(fluid) + (1,) * (3 - len(fluid))
    return {"entry": entry, "dim": dim, "form": form, "fx": fx, "fy": fy, "fz": fz, "steps": steps, "mu": mu,
            "two": two, "tension": tension, "lid": lid, "count": count, "tol": 1e-6 if form == "fp64" else tol}


def listed():
    return [
        # the largest 3D tank of the benchmark (1.3 million particles): a production run
        dict(name="tank3d_100", **_case("advance", 3, "mixed", (100, 100, 100), 3)),
        # a mid-size 3D tank with uneven, odd sides
        dict(name="tank3d_47", **_case("advance", 3, "mixed", (47, 45, 43), 3)),
        # the smallest 3D size that is served (some ten thousand fluid particles): latency counts
        dict(name="tank3d_20", **_case("advance", 3, "mixed", (20, 20, 20), 3)),
        # the 2D dam (10^4 fluid particles), one small case on its own
        dict(name="dam2d_100", **_case("advance", 2, "mixed", (100, 100), 3)),
        # the largest 2D size that is served, two fluids, more viscous
        dict(name="dam2d_613", **_case("advance", 2, "mixed", (613, 651), 2, mu=0.3, two=True)),
        # two fluids with surface tension under a moving, turning lid: the explicit forces and the wall terms
        dict(name="tension3d_33", **_case("advance", 3, "mixed", (37, 29, 33), 2, two=True, tension=0.072, lid=True)),
        # the plain form of the reference's algorithm: small 2D and mid-size 3D
        dict(name="fp64_dam2d_100", **_case("advance", 2, "fp64", (100, 100), 1)),
        dict(name="fp64_tank3d_60", **_case("advance", 3, "fp64", (60, 60, 60), 1)),
        # an output step: every field of a frame after the step (refined further: the pressure is read off the divergence)
        dict(name="frame3d_60", **_case("frame", 3, "mixed", (60, 60, 60), 1, tol=1e-11)),
        # an ensemble of 2D cases of 40 to 250 cells a side, stepped together
        dict(name="ensemble2d_64", **_case("batch", 2, "mixed", (40, 250), 1, count=64)),
        # a short request from its creation to its end
        dict(name="job3d_24", **_case("job", 3, "mixed", (24, 25, 23), 4)),
    ]


def draw(rng):
    entry = rng.choices(["advance", "frame", "batch", "job"], [6, 1, 1, 1])[0]
    if entry == "batch":
        lo = rng.randint(40, 90)
        return _case("batch", 2, "mixed", (lo, rng.randint(lo + 20, 250)), 1, count=rng.randint(6, 48))
    dim = rng.choice([2, 3, 3])
    form = "fp64" if entry == "advance" and rng.random() < 0.25 else "mixed"
    most = {"advance": 700_000, "frame": 250_000, "job": 60_000}[entry]
    if form == "fp64":
        most = 200_000
    if dim == 2:
        most = min(most, 400_000)
    total = math.exp(rng.uniform(math.log(1_500), math.log(most)))      # fluid particles
    side = total ** (1.0 / dim)
    fluid = [max(8, int(round(side * rng.uniform(0.85, 1.15)))) for _ in range(dim)]
    mu = 10.0 ** rng.uniform(-2.0, 0.0 if dim == 2 else -0.5)
    tension = 0.072 if rng.random() < 0.2 else 0.0
    return _case(entry, dim, form, fluid, rng.randint(1, 3), mu=mu, two=rng.random() < 0.4, tension=tension,
                 lid=rng.random() < 0.2, tol=1e-11 if entry == "frame" else 1e-10)


# ---- inputs ----------------------------------------------------------------------
def _one(case, fluid, seed):
    """(params, particles) of one case from the seed alone."""
    dim = case["dim"]
    l0, dt = (0.01, 1e-4) if dim == 2 else (0.005, 5e-5)
    n = fluid[:dim]
    if dim == 2:
        inner = (2 * n[0], int(round(1.5 * n[1])) + 2)
    else:
        inner = tuple(max(k + 2, int(round(a * k))) for a, k in zip((1.6, 1.1, 1.1), n))
    types = None
    if case["two"]:
        up = np.arange(n[-1]) >= n[-1] // 2      # lattice order: the last axis runs fastest
        types = np.tile(up, int(np.prod(n[:-1]))).astype(np.int32)
    top = inner[-1]
    wall = (lambda c: np.where(c[:, dim - 1] >= top, 3, 2)) if case["lid"] else None
    parts = casegen.dam_case(dim, n, inner, l0, seed=seed, fluid_types=types, wall_type_fn=wall)
    params = casegen.baseline_params(dim, l0, dt, mu=case["mu"])
    if case["two"]:
        params = dataclasses.replace(params, density=(1000.0, 1200.0, 1000.0, 1000.0),
                                     interaction_ratio=((1.0, 0.9, 1.0, 1.0), (0.9, 1.0, 1.0, 1.0), (1.0,) * 4, (1.0,) * 4))
    if case["tension"]:
        params = dataclasses.replace(params, surface_tension=(case["tension"], 0.7 * case["tension"], 0.0, 0.0))
    if case["lid"]:
        centre = [0.5 * k * l0 for k in inner] + [0.0] * (3 - dim)
        params = dataclasses.replace(params, wall3=(*centre, 0.05, 0.0, 0.0, 0.0, 0.0, 2.0 if dim == 2 else 0.5))
    rng = np.random.default_rng(seed + 77)
    nf = int(np.prod(n))
    x = parts.pos[:nf]
    a, b = 0, dim - 1                                             # the vortex turns in the plane of x and the vertical
    la, lb = n[a] * l0, n[b] * l0
    u = rng.uniform(0.2, 0.3) * math.sqrt(9.8 * lb)
    ka, kb = math.pi * x[:, a] / la, math.pi * x[:, b] / lb
    parts.vel[:nf, a] = u * np.sin(ka) * np.cos(kb)
    parts.vel[:nf, b] = -u * (lb / la) * np.cos(ka) * np.sin(kb)
    parts.vel[:nf, :dim] += rng.uniform(-1e-3 * u, 1e-3 * u, size=(nf, dim))
    return params, parts


def _inputs(case, seed):
    """[(params, particles)] of the case: one, or `count` of a batch."""
    if case["entry"] != "batch":
        return [_one(case, (case["fx"], case["fy"], case["fz"]), seed)]
    rng = np.random.default_rng(1)      # the sizes belong to the case, what fills them to the seed
    got = []
    for k in range(case["count"]):
        n, m = (int(v) for v in rng.integers(case["fx"], case["fy"] + 1, size=2))
        sub = dict(case, two=k % 2 == 1, mu=float(10.0 ** rng.uniform(-2.0, 0.0)))
        got.append(_one(sub, (n, m, 1), seed * 1000003 + k))
    return got


def _pinned(shape, dtype):
    t = torch.empty(shape, dtype={np.float64: torch.float64, np.int32: torch.int32}[dtype], pin_memory=torch.cuda.is_available())
    return t.numpy()


FRAME = (("id", np.int32, 0), ("type", np.int32, 0), ("neighbor_count", np.int32, 0), ("pos", np.float64, 3), ("vel", np.float64, 3),
         ("force", np.float64, 3), ("vol_strain_p", np.float64, 0), ("divergence_p", np.float64, 0),
         ("pressure_p", np.float64, 0), ("virial_p", np.float64, 0))
STATE = tuple(f for f in FRAME if f[0] in ("id", "type", "pos", "vel"))


def _new(case, params, parts):
    c = engine.Case(params, parts, case["dim"], precision=PRECISION_MIXED if case["form"] == "mixed" else PRECISION_FP64)
    if case["form"] == "mixed":
        c.set_solver(case["tol"], 1e-3, 50)
        c.set_option("extrapolate", 2)
    return c


def prepare(case, seed):
    made = _inputs(case, seed)
    ups, total = [], sum(p.count for _, p in made)
    out = {k: _pinned((total, w) if w else (total,), t) for k, t, w in (FRAME if case["entry"] == "frame" else STATE)}
    views, at = [], 0
    for params, parts in made:
        n = parts.count
        up = casegen.Particles(parts.time, parts.spacing, parts.domain_min, parts.domain_max, _pinned((n,), np.int32),
                               _pinned((n, 3), np.float64), _pinned((n, 3), np.float64))
        up.types[:], up.pos[:], up.vel[:] = parts.types, parts.pos, parts.vel
        ids = _pinned((n,), np.int32)
        ids[:] = np.arange(n)
        ups.append((params, up, ids, np.zeros((4, 3))))
        ups[-1][3][2], ups[-1][3][3] = params.wall2[:3], params.wall3[:3]
        views.append({k: a[at:at + n] for k, a in out.items()})
        at += n
    cases = [] if case["entry"] == "job" else [_new(case, p, u) for p, u, _, _ in ups]
    return {"case": case, "ups": ups, "cases": cases, "views": views, "out": out}


def run(state):
    case, ups, cases, views = state["case"], state["ups"], state["cases"], state["views"]
    if case["entry"] == "job":
        params, up, _, _ = ups[0]
        c = _new(case, params, up)
        c.step(case["steps"])
        c.fields(out=views[0])
        c.close()
        return state["out"]
    for c, (_, up, ids, centre) in zip(cases, ups):
        c.set_state(up, ids, centre)
    if case["entry"] == "batch":
        engine.batch_step(cases, case["steps"])
    else:
        cases[0].step(case["steps"])
    for c, v in zip(cases, views):
        if case["entry"] == "frame":
            c.stage("output_fields")
        c.fields(out=v)
    return state["out"]


# ---- work ------------------------------------------------------------------------
def work(case):
    """The state read and written once; the arithmetic of the step: for every particle the weights of its neighbours,
    for every iteration of the linear solve (about 100) the products with C, its transpose and the viscous pairs."""
    if case["entry"] == "batch":
        side = 0.5 * (case["fx"] + case["fy"])
        nf, n = case["count"] * side * side, case["count"] * (side * side + 24 * side)
    else:
        nf = case["fx"] * case["fy"] * case["fz"]
        n = 1.3 * nf if case["dim"] == 3 else nf + 24 * math.sqrt(nf)
    d, nb, npl = case["dim"], (37 if case["dim"] == 2 else 179), (9 if case["dim"] == 2 else 19)
    words = 2 * 48 + 2 * 8 if case["entry"] != "frame" else 48 + 8 + 3 * 24 + 4 * 8 + 3 * 4
    per = n * nb * 12 + nf * nb * 8 * d + 100 * nf * (npl * 4 * d + nb * 4 * d + 14 * d)
    return {"bytes": float(n * words), "flops": float(case["steps"] * per)}


# ---- the step in 64 bits ---------------------------------------------------------
def _quad(kf, r, h):
    return kf * (1.0 - r / h) ** 2


def _dquad(kf, r, h):
    return kf * (-2.0 / h) * (1.0 - r / h)


class _Step:
    """The method's constants and one time step of it on torch tensors (particles in the order of the input)."""

    def __init__(self, p, parts, dim, device):
        self.p, self.dim, self.dev = p, dim, device
        l0 = parts.spacing
        self.l0, self.vol, self.dt = l0, l0 ** dim, p.dt
        self.rA, self.rP, self.rV = p.radius_ratio_a * l0, p.radius_ratio_p * l0, p.radius_ratio_v * l0
        self.rG = self.rA
        if dim == 2:
            swa, swg = 1 / 2 * 2 / 15 * math.pi / l0 / l0, 1 / 2 * 1 / 3 * math.pi / l0 / l0
            self.R2g = 1 / 2 * 1 / 30 * math.pi * self.rG * self.rG / l0 / l0 / swg
            self.cofK, integN, integX, self.visc = 0.350778153, 0.024679383, 0.226126699, 8.0
        else:
            swa, swg = 1 / 3 * 1 / 5 * math.pi / l0 ** 3, 1 / 3 * 2 / 5 * math.pi / l0 ** 3
            self.R2g = 1 / 3 * 4 / 105 * math.pi * self.rG * self.rG / l0 ** 3 / swg
            self.cofK, integN, integX, self.visc = 0.326976006, 0.021425779, 0.233977488, 10.0
        self.kfa, self.kfg = (1 / swa) / self.rA ** dim, (1 / swg) / self.rG ** dim
        self.kfp, self.kfv = (1 / swg) / self.rP ** dim, (1 / swg) / self.rV ** dim
        self.N0a, self.N0p = self._lattice(self.rA, True), self._lattice(self.rP, False)
        t = lambda v: torch.tensor(v, dtype=torch.float64, device=device)  # noqa: E731
        self.cofA = t([s / ((self.rG / l0) * (integN + self.cofK ** 2 * integX)) for s in p.surface_tension])
        self.rho, self.bulk, self.lam, self.mu = t(p.density), t(p.bulk_modulus), t(p.bulk_viscosity), t(p.shear_viscosity)
        self.ratio = t(p.interaction_ratio)
        self.maxR = max(self.rA, 2.0 * self.rP, self.rV)
        self.lo = [float(v) for v in parts.domain_min[:dim]]
        self.W = [float(b) - float(a) for a, b in zip(parts.domain_min[:dim], parts.domain_max[:dim])]
        self.cc = [int(math.floor(w / self.maxR)) for w in self.W]
        # as tensors: a quotient by a plain number is rounded as a product with its reciprocal on a GPU
        self.cwt, self.Wt = t([w / c for w, c in zip(self.W, self.cc)]), t(self.W)
        self.T = int(np.prod(self.cc))
        self.walls = {2: np.array(p.wall2, float), 3: np.array(p.wall3, float)}
        self.centre = {k: w[:3].copy() for k, w in self.walls.items()}

    def _lattice(self, h, a):
        k = int(math.ceil(h / self.l0))
        ax = np.arange(-k, k + 1) * self.l0
        g = np.meshgrid(*([ax] * self.dim), indexing="ij")
        r2 = sum(v * v for v in g).ravel()
        q = np.sqrt(r2[(r2 > 0) & (r2 <= h * h)]) / h
        return float(np.sum(self.kfa * q * (1 - q) ** 2 if a else self.kfp * (1 - q) ** 2))

    def keys(self, x, typ):
        k = torch.zeros(len(x), dtype=torch.int64, device=self.dev)
        for d in range(self.dim):
            k = k * self.cc[d] + torch.floor((x[:, d] - self.lo[d]) / self.cwt[d]).long() % self.cc[d]
        return k + torch.where(typ >= 2, self.T, 0)

    def sort(self, x, typ):
        """The order after the method's sort: its compare-exchange network on the cell keys (it is not stable)."""
        n = len(x)
        e = n.bit_length()
        key = torch.full((1 << e,), 2 * self.T, dtype=torch.int64, device=self.dev)
        key[:n] = self.keys(x, typ)
        perm = torch.arange(1 << e, device=self.dev)
        at = torch.arange(1 << e, device=self.dev)
        for m in range(e):
            for s in range(m + 1):
                d = 1 << (m - s)
                i = at[(at & d) == 0]
                j = i | d
                up = ((i >> m) & 2) == 0
                ki, kj, pi, pj = key[i], key[j], perm[i], perm[j]
                sw = (ki > kj) == up
                key[i], key[j] = torch.where(sw, kj, ki), torch.where(sw, ki, kj)
                perm[i], perm[j] = torch.where(sw, pj, pi), torch.where(sw, pi, pj)
        return perm[:n]

    def sep(self, x, i, j):
        q = x[j] - x[i]
        for d in range(self.dim):
            t = q[:, d] + 0.5 * self.W[d]
            q[:, d] = (t - self.W[d] * torch.floor(t / self.Wt[d])) - 0.5 * self.W[d]
        return q

    def pairs(self, x, typ):
        n, dev = len(x), self.dev
        cell = [torch.floor((x[:, d] - self.lo[d]) / self.cwt[d]).long() % self.cc[d] for d in range(self.dim)]
        flat = torch.zeros(n, dtype=torch.int64, device=dev)
        for d in range(self.dim):
            flat = flat * self.cc[d] + cell[d]
        order = torch.argsort(flat)
        cnt = torch.bincount(flat, minlength=self.T)
        start = torch.cumsum(cnt, 0) - cnt
        I, J = [], []
        for o in np.ndindex(*([3] * self.dim)):
            nb = torch.zeros(n, dtype=torch.int64, device=dev)
            for d in range(self.dim):
                nb = nb * self.cc[d] + (cell[d] + o[d] - 1) % self.cc[d]
            c = cnt[nb]
            i = torch.repeat_interleave(torch.arange(n, device=dev), c)
            first = torch.cumsum(c, 0) - c
            j = order[start[nb][i] + torch.arange(len(i), device=dev) - first[i]]
            keep = (self.sep(x, i, j) ** 2).sum(1) <= self.maxR ** 2
            keep &= i != j
            I.append(i[keep])
            J.append(j[keep])
        i, j = torch.cat(I), torch.cat(J)
        # a wall particle without fluid neighbours has no neighbours at all
        wet = torch.zeros(n, dtype=torch.bool, device=dev)
        wet[i[typ[j] < 2]] = True
        keep = (typ[i] < 2) | wet[i]
        return i[keep], j[keep]

    def move(self, x, v, typ):
        dt = self.dt
        fl = typ < 2
        x = torch.where(fl[:, None], x + v * dt, x)
        for t, w in self.walls.items():
            me = typ == t
            vel, om = w[3:6], w[6:9]
            th = abs(float(om @ om))
            ax = om / th if th else np.zeros(3)
            s, q3 = math.sin(th * dt / 2), math.cos(th * dt / 2)
            q0, q1, q2 = ax * s
            R = np.array([[q0 * q0 - q1 * q1 - q2 * q2 + q3 * q3, 2 * (q0 * q1 - q2 * q3), 2 * (q0 * q2 + q1 * q3)],
                          [2 * (q0 * q1 + q2 * q3), -q0 * q0 + q1 * q1 - q2 * q2 + q3 * q3, 2 * (q1 * q2 - q0 * q3)],
                          [2 * (q0 * q2 - q1 * q3), 2 * (q1 * q2 + q0 * q3), -q0 * q0 - q1 * q1 + q2 * q2 + q3 * q3]])
            c = self.centre[t]
            r = [x[me, d] - c[d] if d < self.dim else torch.zeros_like(x[me, 0]) for d in range(3)]
            for a in range(3):   # rotated in place, component by component
                r[a] = R[a, 0] * r[0] + R[a, 1] * r[1] + R[a, 2] * r[2]
            u = [om[1] * r[2] - om[2] * r[1] + vel[0], om[2] * r[0] - om[0] * r[2] + vel[1], om[0] * r[1] - om[1] * r[0] + vel[2]]
            v, x = v.clone(), x.clone()
            for d in range(self.dim):
                v[me, d] = u[d]
                x[me, d] = (r[d] + c[d]) + vel[d] * dt
            self.centre[t] = c + vel * dt
        for d in range(self.dim):
            t = x[:, d] - self.lo[d]
            x[:, d] = (t - self.W[d] * torch.floor(t / self.Wt[d])) + self.lo[d]
        return x, v

    def step(self, x, v, typ, ids):
        x, v = self.move(x.clone(), v.clone(), typ)
        o = self.sort(x, typ)
        x, v, typ, ids = x[o], v[o], typ[o], ids[o]
        n, D = len(x), self.dim
        nf = int((typ < 2).sum())
        i, j = self.pairs(x, typ)
        q = self.sep(x, i, j)
        r = q.pow(2).sum(1).sqrt()
        e = q / r[:, None]
        ti, tj = typ[i], typ[j]
        zero = torch.zeros(n, dtype=torch.float64, device=self.dev)
        add = lambda at, w, like=zero: torch.zeros_like(like).index_add_(0, at, w)  # noqa: E731
        zv = torch.zeros_like(x)
        self.i, self.j, self.q, self.r, self.e = i, j, q, r, e
        inP, inA, inV = r <= self.rP, r <= self.rA, r < self.rV
        P = torch.nonzero(inP).ravel()
        pi, pj = i[P], j[P]
        vsp = add(pi, _quad(self.kfp, r[P], self.rP)) - self.N0p
        rij, rji = self.ratio[ti, tj], self.ratio[tj, ti]
        h = r / self.rA
        wa = torch.where(inA, self.kfa * h * (1 - h) ** 2, 0.0)
        wg = torch.where(inA, _quad(self.kfg, r, self.rG), 0.0)
        gcen = add(i, q * (rij * wg)[:, None] / self.R2g * self.rG, zv)
        densA = add(i, rij * wa)
        presA = torch.where(densA >= self.N0a, 0.0, self.cofA[typ] * (densA - self.N0a) / self.l0)
        force = zv.clone()
        if bool((self.cofA != 0).any()):
            dwa = torch.where(inA, self.kfa * (1 - h) * (1 - 3 * h) / self.rA, 0.0)
            dwg = torch.where(inA, _dquad(self.kfg, r, self.rG), 0.0)
            fa = (presA[i] * rij + presA[j] * rji) * dwa * self.vol
            k = self.cofA[ti] * self.cofK ** 2
            sc = self.rG * self.vol / self.l0 / self.R2g
            gi, gj = gcen[i], gcen[j]
            f = fa[:, None] * e - (k * sc)[:, None] * (gj * (rji * wg)[:, None] - gi * (rij * wg)[:, None])
            gr = ((gj * (rji * dwg)[:, None] - gi * (rij * dwg)[:, None]) * q).sum(1) * k * sc
            force = add(i, f - gr[:, None] * e, zv)
        g = torch.tensor(self.p.gravity[:D], dtype=torch.float64, device=self.dev)
        m = (self.rho[typ] * self.vol)[:, None]
        fl = (typ < 2)[:, None]
        force = torch.where(fl, force + m * g, force)
        start = v[:nf].clone()
        v = torch.where(fl, v + force / m * self.dt, v)
        # the implicit system of the fluid rows
        wd = -_dquad(self.kfv, r, self.rV)
        mu = self.mu
        V = torch.nonzero((ti < 2) & inV).ravel()
        mui, muj = mu[ti[V]], mu[tj[V]]
        f = self.visc * (2 * mui * muj / (mui + muj)) * wd[V] / r[V]
        vi, vj, ve = i[V], j[V], e[V]
        wet = (tj[V] < 2)[:, None]
        cw = -_dquad(self.kfp, r[P], self.rP)
        inside = (r[P] < self.rP)
        cw = torch.where(inside, cw, 0.0)
        ce = e[P] * cw[:, None]
        R = torch.nonzero(ti[P] < 2).ravel()
        ci, ck, cv = pi[R], pj[R], ce[R]
        cs = add(ci, cv, zv)                                       # the row's own entry of C
        lam = self.lam[typ]
        pvec = torch.where(vsp > 0, self.bulk[typ] * vsp, 0.0)
        wi, wj = (ti[P] >= 2)[:, None], (tj[P] >= 2)[:, None]
        pvec = pvec + add(pi, lam[pi] * (torch.where(wi, ce * v[pi], 0.0) - torch.where(wj, ce * v[pj], 0.0)).sum(1))
        inert = (self.rho[typ] / self.dt)[:nf, None]
        fe = f[:, None] * ve
        b = add(vi, torch.where(wet, 0.0, fe * (ve * v[vj]).sum(1)[:, None]), zv)
        b = b - add(ci, cv * pvec[ck][:, None], zv) - cs * pvec[:, None]
        b = b[:nf] + inert * v[:nf]

        def A(u):
            full = torch.zeros_like(x)
            full[:nf] = u
            d = full[vi] - torch.where(wet, full[vj], 0.0)
            y = add(vi, fe * (ve * d).sum(1)[:, None], zv)
            t = lam * (add(ck, (cv * full[ci]).sum(1)) + (cs * full).sum(1))
            return inert * u + y[:nf] + (add(ci, cv * t[ck][:, None], zv) + cs * t[:, None])[:nf]

        diag = inert + (add(vi, fe * ve, zv) + add(ci, cv * cv * lam[ck][:, None], zv) + cs * cs * lam[:, None])[:nf]
        u = start
        res = b - A(u)
        z = res / diag
        d = z
        rz = (res * z).sum()
        stop = 1e-14 * float(b.norm())
        for it in range(600):
            Ad = A(d)
            al = rz / (d * Ad).sum()
            u = u + al * d
            res = res - al * Ad
            if it % 10 == 9 and float(res.norm()) < stop:
                break
            z = res / diag
            new = (res * z).sum()
            d = z + (new / rz) * d
            rz = new
        v = v.clone()
        v[:nf] = u
        self.last = dict(vsp=vsp, gcen=gcen, presA=presA, P=P, ce=ce, lam=lam)
        return x, v, typ, ids, force

    def frame(self, x, v, typ, force):
        """The fields of an output frame: divergence, pressure, the forces and the virial pressure."""
        L = self.last
        i, j, q, r, e, P, lam = self.i, self.j, self.q, self.r, self.e, L["P"], L["lam"]
        n, D, zv = len(x), self.dim, torch.zeros_like(x)
        zero = torch.zeros(n, dtype=torch.float64, device=self.dev)
        add = lambda at, w, like=zero: torch.zeros_like(like).index_add_(0, at, w)  # noqa: E731
        pi, pj = i[P], j[P]
        dw = _dquad(self.kfp, r[P], self.rP)
        div = -add(pi, ((v[pj] - v[pi]) * e[P]).sum(1) * dw)
        pres = -lam * div + torch.where(L["vsp"] > 0, self.bulk[typ] * L["vsp"], 0.0)
        fp = add(pi, ((pres[pi] + pres[pj]) * dw)[:, None] * e[P] * self.vol, zv)
        inV = r < self.rV
        ti, tj = typ[i], typ[j]
        mui, muj = self.mu[ti], self.mu[tj]
        fv = self.visc * 2 * mui * muj / (mui + muj) * ((v[j] - v[i]) * e).sum(1) * -_dquad(self.kfv, r, self.rV) / r * self.vol
        fv = torch.where(inV, fv, 0.0)[:, None] * e
        tr = add(pi, pres[pi] * dw * r[P]) + add(i, 0.5 * (fv * q).sum(1) / self.vol)
        inA = r < self.rA
        h = r / self.rA
        rij = self.ratio[ti, tj]
        tr = tr + add(i, torch.where(inA, L["presA"][i] * rij * self.kfa * (1 - h) * (1 - 3 * h) / self.rA * r, 0.0))
        a = self.cofA[ti] * self.cofK ** 2
        gq = (-L["gcen"][i] * q).sum(1)
        s = -a * gq * rij * (_quad(self.kfg, r, self.rG) + _dquad(self.kfg, r, self.rG) * r) / self.R2g * self.rG / self.l0
        tr = tr + add(i, torch.where(inA, s, 0.0))
        return {"force": force + fp + add(i, fv, zv), "vol_strain_p": L["vsp"], "divergence_p": div, "pressure_p": pres,
                "virial_p": -tr / D}


def exact(case, seed):
    made = _inputs(case, seed)
    if sum(p.count for _, p in made) * max(1.0, case["steps"] / 2) > EXACT_MAX * (6 if case["dim"] == 2 else 1):
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    got = []
    for params, parts in made:
        S = _Step(params, parts, case["dim"], dev)
        t = lambda a: torch.from_numpy(np.array(a)).to(dev)  # noqa: E731
        x, v, typ, ids = t(parts.pos[:, :S.dim]), t(parts.vel[:, :S.dim]), t(parts.types).long(), torch.arange(parts.count, device=dev)
        if case["entry"] == "job":      # a new case sorts its particles once before the first step
            o = S.sort(x, typ)
            x, v, typ, ids = x[o], v[o], typ[o], ids[o]
        for _ in range(case["steps"]):
            x, v, typ, ids, force = S.step(x, v, typ, ids)
        f = {"pos": x, "vel": v}
        if case["entry"] == "frame":
            f.update(S.frame(x, v, typ, force))
        for k, a in f.items():
            if a.dim() == 2 and S.dim == 2:     # the z of the plane is 0
                f[k] = torch.cat([a, torch.zeros_like(a[:, :1])], 1)
        got.append(f)
    whole = {k: None for k, _, _ in (FRAME if case["entry"] == "frame" else STATE)}
    whole.update({k: torch.cat([f[k] for f in got]) for k in got[0]})
    return whole
