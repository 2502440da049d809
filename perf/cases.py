"""The work that a user of the engine has it do, as cases to be timed and compared.

Most cases are one RK2 cycle (two stages and the dt policy) of a job, replayed
from its captured graph as ``Simulation.step`` and ``Pool.step`` do it; one
goes task by task over pointer tables, as a Parthenon build drives the engine.
``exact`` restates the stage in plain torch FP64, from the inputs that
``prepare`` made and from nothing else of this repository.
"""
from __future__ import annotations

import math
import random

import torch

from pangu_b200 import problems
from pangu_b200.engine import RK2_BETA, Engine, Pool, Simulation, TableContainer
from pangu_b200.params import mesh_struct, params_struct, process_packages

DEV = "cuda:0"
PERIODIC, OUTFLOW = 0, 1


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def _case(kind, problem, nx, block=None, precision="fp64", limiter="ppm4", riemann="laxf",
          recovery="chainer", heating="constant", metric="mks", settle=20, jobs=1):
    bx = block or nx
    return {"kind": kind, "problem": problem, "nx1": nx[0], "nx2": nx[1], "nx3": nx[2],
            "bx1": bx[0], "bx2": bx[1], "bx3": bx[2], "precision": precision,
            "limiter": limiter, "riemann": riemann, "recovery": recovery, "heating": heating,
            "metric": metric, "settle": settle, "jobs": jobs}


def listed():
    named = {
        # the smallest job: a shock tube, where launches and latency are the time
        "bw_1024_fp64": _case("cycle", "bw", (1024, 1, 1), limiter="mc", riemann="hll",
                              metric="minkowski"),
        # a ragged vortex (rows of an odd length) in the mixed form
        "ot_129_mixed": _case("cycle", "ot", (129, 129, 1), precision="mixed", limiter="mc",
                              heating="", metric="minkowski"),
        # the Orszag-Tang benchmark
        "ot_256_fp64": _case("cycle", "ot", (256, 256, 1), limiter="mc", heating="",
                             metric="minkowski"),
        # a large flat-space run, with the dearer options
        "ot_1024_ppm4_hll_fp64": _case("cycle", "ot", (1024, 1024, 1), riemann="hll",
                                       metric="minkowski"),
        # the torus benchmark in both precisions
        "torus_512x256_fp64": _case("cycle", "torus", (512, 256, 1)),
        "torus_512x256_mixed": _case("cycle", "torus", (512, 256, 1), precision="mixed"),
        # first cycles of a small odd torus in Boyer-Lindquist coordinates, when
        # many cells fail the first inversion scheme; an exp/log heating model
        "torus_bl_201x99_fp64": _case("cycle", "torus", (201, 99, 1), heating="howes",
                                      metric="bl", settle=3),
        # production: the torus in three dimensions, several meshblocks
        "torus3d_fp64": _case("cycle", "torus", (256, 128, 128), (64, 64, 64), riemann="hll"),
        "torus3d_mixed": _case("cycle", "torus", (256, 128, 128), (64, 64, 64), riemann="hll",
                               precision="mixed"),
        # an excised hole in Cartesian coordinates: the metric is not tabulated
        "cks_64_fp64": _case("cycle", "cks", (64, 64, 64), (32, 32, 32), limiter="mc",
                             heating="", metric="cks"),
        # many uneven tori stepped together
        "batch_12_fp64": _case("batch", "torus", (128, 64, 1), jobs=12),
        # one stage by single tasks over per-variable allocations, as a
        # Parthenon build calls them; odd sizes, the other solvers
        "tasks_333x127_fp64": _case("tasks", "torus", (333, 127, 1), limiter="mc", riemann="hll",
                                    recovery="robuster", heating="kawazura"),
    }
    return [dict(c, name=n) for n, c in named.items()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    pick = rng.choice
    options = dict(precision=pick(("fp64", "mixed")), limiter=pick(("mc", "ppm4")),
                   riemann=pick(("laxf", "hll")),
                   recovery=pick(("chainer", "chainer", "robuster")),
                   heating=pick(("constant", "constant", "howes", "kawazura", "sharma", "")),
                   settle=pick((3, 8, 20)))
    if options["precision"] == "mixed":
        # the other inversion and the exp/log heating models amplify a 32-bit
        # rounding in the torus' atmosphere until outputs cannot be compared
        options["recovery"] = "chainer"
        if options["heating"] in ("howes", "kawazura"):
            options["heating"] = "constant"
    kind = pick(("bw", "ot", "ot", "torus", "torus", "torus3d", "torus3d", "cks", "batch", "tasks"))
    if kind == "bw":
        return _case("cycle", "bw", (_log_int(rng, 256, 16384), 1, 1), metric="minkowski",
                     **options)
    if kind == "ot":
        n = _log_int(rng, 48, 1024)
        return _case("cycle", "ot", (n, n, 1), metric="minkowski", **options)
    if kind in ("torus", "tasks"):
        nx = (_log_int(rng, 64, 768), _log_int(rng, 32, 384), 1)
        if kind == "tasks":
            options["precision"] = "fp64"
        return _case("cycle" if kind == "torus" else "tasks", "torus", nx,
                     metric=pick(("mks", "mks", "bl")), **options)
    if kind == "torus3d":
        b = (_log_int(rng, 20, 64), _log_int(rng, 16, 64), _log_int(rng, 8, 64))
        m = (rng.randint(1, 3), rng.randint(1, 2), rng.randint(1, 2))
        return _case("cycle", "torus", tuple(x * y for x, y in zip(b, m)), b, **options)
    if kind == "cks":
        b, m = _log_int(rng, 12, 40), rng.randint(1, 2)
        options.update(heating="", limiter="mc")
        return _case("cycle", "cks", (b * m,) * 3, (b,) * 3, metric="cks", **options)
    return _case("batch", "torus", (128, 64, 1), jobs=rng.randint(3, 16), **options)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _options(pin, c, precision):
    ppm4 = c["limiter"] == "ppm4"
    for key in ("limiter", "recovery"):
        pin.set("core", key, c[key])
    pin.set("core", "riemann_solver", c["riemann"])
    pin.set("core", "enable_heating", bool(c["heating"]))
    if c["heating"]:
        pin.set("electron", "model", c["heating"])
    pin.set("parthenon/mesh", "nghost", 3 if ppm4 else 2)
    pin.set("metric", "type", c["metric"])
    if c["metric"] == "bl":  # outside the horizon of these coordinates
        pin.set("parthenon/mesh", "x1min", 0.7)
    pin.set("b200", "precision", precision)
    return pin


def _input(c, seed, precision, nx=None, **torus):
    nx = nx or (c["nx1"], c["nx2"], c["nx3"])
    bx = (c["bx1"], c["bx2"], c["bx3"])
    if c["problem"] == "bw":
        pin = problems.brio_wu_input(n=nx[0], nblock=bx[0])
    elif c["problem"] == "ot":
        pin = problems.orszag_tang_input(n=nx[0], nblock=bx[0])
    elif c["problem"] == "cks":
        pin = problems.cks_atmosphere_input(n=nx[0], nblock=bx[0])
    else:
        pin = problems.fm_torus_input(*nx, bx, seed=seed, **torus)
    return _options(pin, c, precision)


def _shaken(prim, seed):
    """Density and internal energy scaled by 1 + O(0.5 %), different for every seed."""
    g = torch.Generator(device=prim.device).manual_seed(seed)
    u = torch.rand((prim.shape[0], 2) + prim.shape[2:], generator=g, device=prim.device,
                   dtype=torch.float64)
    prim[:, :2] *= 1.0 + 0.01 * (u - 0.5).to(prim.dtype)
    return prim


def _settled(c, seed):
    """A job `settle` cycles from its seeded initial state; the mixed form
    continues from the state that an FP64 job reached."""
    sim = Simulation(_input(c, seed, "fp64"), device=0)
    if c["metric"] in ("cks", "bl"):  # made on the host
        geo = problems.Geometry(sim.mesh)
        prim = torch.as_tensor(problems.cks_atmosphere(geo, sim.packages)
                               if c["problem"] == "cks" else
                               problems.fm_torus(geo, sim.packages, sim.pin), device=DEV)
    else:
        sim.generate(c["problem"])
        prim = sim.base.prim.clone()
    sim.set_primitives(_shaken(prim, seed))
    if c["settle"]:
        sim.capture()
    for _ in range(c["settle"]):
        sim.step()
    if c["precision"] == "fp64":
        sim._graph = None
        return sim
    mixed = Simulation(_input(c, seed, "mixed"), device=0)
    for name in ("base", "one"):
        src, dst = getattr(sim, name), getattr(mixed, name)
        dst.prim.copy_(src.prim)
        dst.cons.copy_(src.cons)
    mixed.base.flag.copy_(sim.base.flag)
    mixed.dt.copy_(sim.dt)
    if not c["settle"]:
        mixed.set_primitives(prim)
    torch.cuda.synchronize()
    return mixed


BATCH_GRIDS = ((128, 64), (256, 128), (384, 192), (512, 256))


def _fields(c, prim):
    """The primitive variables by name; a vector is one output, since a
    component that vanishes in the continuum holds only rounding noise."""
    parts = {"density": (0, 1), "energy": (1, 2), "velocity": (2, 5), "field": (5, 8),
             "entropy": (8, 9)}
    if c["heating"]:
        parts["electron_entropy"] = (9, 10)
    return {n: prim[:, a:b] for n, (a, b) in parts.items()}


def _outputs(c, base, one, dt):
    out = _fields(c, base.prim)
    out.update(one_prim=one.prim, base_cons=base.cons, one_cons=one.cons, dt=dt)
    if c["recovery"] == "chainer":
        out["flag"] = base.flag
    return out


def prepare(case, seed):
    c = case
    if c["kind"] == "batch":
        rng = random.Random(seed)
        pins = []
        for q in range(c["jobs"]):
            nx = BATCH_GRIDS[q % len(BATCH_GRIDS)] + (1,)
            pins.append(_input(c, seed * 64 + q, "fp64", nx, a=rng.uniform(0.5, 0.95),
                               rmax=rng.uniform(11.0, 13.0),
                               beta=math.exp(rng.uniform(math.log(30.0), math.log(300.0)))))
        blocks = sum(_blocks(p) for p in pins)

        def fill(precision, states=None):
            pool = Pool(_options(pins[0], c, precision), blocks, len(pins), device=0)
            for q, pin in enumerate(pins):
                _options(pin, c, precision)
                if states is None:
                    pool.attach_problem(pin, "torus")
                else:
                    pool.attach(pin, states[q])
            return pool

        pool = fill("fp64")
        for _ in range(c["settle"]):
            pool.step()
        if c["precision"] == "mixed":
            old, pool = pool, fill("mixed", [p for p in _per_job(pool)])
            for name in ("base", "one"):
                src, dst = getattr(old, name), getattr(pool, name)
                if c["settle"]:
                    dst.prim.copy_(src.prim)
                    dst.cons.copy_(src.cons)
            pool.base.flag.copy_(old.base.flag)
            pool.dt.copy_(old.dt)
        pool.autotune()
        torch.cuda.synchronize()
        return {"pool": pool, "pins": pins, "out": _outputs(c, pool.base, pool.one, pool.dt)}
    sim = _settled(c, seed)
    if c["kind"] == "cycle":
        sim.autotune()
        sim.capture()
        torch.cuda.synchronize()
        return {"sim": sim, "out": _outputs(c, sim.base, sim.one, sim.dt)}
    # stage tasks over one allocation per block and variable
    e = Engine(sim.params, sim.mesh, 0)
    groups = (1, 1, 3, 3, 1) + ((1,) if c["heating"] else ())
    base = TableContainer(e.nb, e.nf, e.shape, e.device, prim_groups=groups, cons_groups=(e.nf,))
    one = TableContainer(e.nb, e.nf, e.shape, e.device, prim_groups=groups, cons_groups=(e.nf,),
                         shared=base)
    base.load(sim.base)
    one.load(sim.one)
    est = torch.zeros(1, dtype=torch.float64, device=DEV)
    out = {"base_prim": base.arrays["prim"][0], "one_prim": one.arrays["prim"][0],
           "base_cons": base.arrays["cons"][0], "one_cons": one.arrays["cons"][0], "dt": est}
    if c["recovery"] == "chainer":
        out["flag"] = base.arrays["flag"][0]
    torch.cuda.synchronize()
    return {"engine": e, "base": base, "one": one, "dt": sim.dt.clone(), "est": est,
            "pin": sim.pin, "out": out}


def _blocks(pin):
    m = mesh_struct(pin)
    return m.nbx1 * m.nbx2 * m.nbx3


def _per_job(pool):
    for slots in pool.jobs.values():
        yield pool.base.prim[torch.tensor(slots, device=DEV)].clone()


def run(state):
    if "sim" in state:
        state["sim"].step()
        return state["out"]
    if "pool" in state:
        state["pool"].step()
        return state["out"]
    e, base, one, dt = state["engine"], state["base"], state["one"], state["dt"]
    e.fix_primitive(base)
    e.calculate_conservative(base)
    e.calculate_fluxes(base)
    e.constrained_transport(base)
    e.flux_divergence_update(base, base, one, RK2_BETA[1], dt)
    e.exchange_ghosts(one)
    e.add_geometric_source(one, RK2_BETA[1], dt)
    e.recovery(one)
    e.apply_electron_heating(one)
    if e.params.recovery == 0:
        e.fix_recovery(one)
    e.apply_boundary_conditions(one)
    e.estimate_dt(one, state["est"])
    return state["out"]


def work(case):
    """Per cell and stage: both containers' primitives read and one written,
    one container's conserved variables written, flags; operations of the
    stage's formulas (reconstruction, two states and a flux per face, the
    inversion's Newton steps, the rest), counted by hand."""
    c = case
    cells = c["nx1"] * c["nx2"] * c["nx3"]
    if c["kind"] == "batch":
        cells = sum(a * b for q in range(c["jobs"]) for a, b in [BATCH_GRIDS[q % 4]])
    nf = 10 if c["heating"] else 9
    p = 8 if c["precision"] == "fp64" else 4
    ndim = 1 + (c["nx2"] > 1) + (c["nx3"] > 1)
    curved = c["metric"] != "minkowski"
    face = 10 * (30 if c["limiter"] == "ppm4" else 12) + (620 if curved else 420)
    flops = ndim * face + 5 * 70 + 150 + (450 if curved else 150) + 12 * nf * ndim
    stages = 1 if c["kind"] == "tasks" else 2
    return {"bytes": float(cells * stages * (nf * (2 * p + p + 8) + 16)),
            "flops": float(cells * stages * flops)}


def tolerance(case):
    # The FP64 form gives the same bits on every build: the inversion chain is
    # chaotic in its last bits, and the oracle tests ask for them. The mixed
    # form's primitives, fluxes and sources are 32-bit numbers; measured
    # against exact(), its outputs are up to 2e-5 off (3e-3 in single cells,
    # where the inversion amplifies a rounding).
    if case["precision"] == "fp64":
        return "exact"
    return {"rel": 1e-4, "max": 0.05, "differ": 1e-3}


# ---------------------------------------------------------------------------
# The stage in plain torch, FP64
# ---------------------------------------------------------------------------
def _det3(a, b, c, d, e, f, g, h, i):
    return a * (e * i - f * h) - b * (d * i - f * g) + c * (d * h - e * g)


def _inverse(g):
    """(inverse, determinant) of a 4 x 4 matrix of tensors."""
    rows = range(4)

    def minor(r, c):
        rr, cc = [x for x in rows if x != r], [x for x in rows if x != c]
        return _det3(*[g[i][j] for i in rr for j in cc])

    cof = [[(-1) ** (r + c) * minor(r, c) for c in rows] for r in rows]
    det = sum(g[0][c] * cof[0][c] for c in rows)
    return [[cof[c][r] / det for c in rows] for r in rows], det


def _where(m, a, b):
    return torch.where(m, torch.as_tensor(a, device=m.device, dtype=torch.float64),
                       torch.as_tensor(b, device=m.device, dtype=torch.float64))


RHO, ENY, U1, B1, ENT, KEL = 0, 1, 2, 5, 8, 9


class _Stage:
    """One job's mesh, metric and tasks on arrays [block][variable][k][j][i]."""

    def __init__(self, pin, mixed, dev):
        pk = process_packages(pin)
        self.p, self.m, self.mixed, self.dev = params_struct(pk), mesh_struct(pin), mixed, dev
        self.c, self.mt = pk["core"].params, pk["metric"].params["metric_type"]
        m = self.m
        self.bx, self.lat = (m.nx1, m.nx2, m.nx3), (m.nbx1, m.nbx2, m.nbx3)
        self.nb = m.nbx1 * m.nbx2 * m.nbx3
        self.act = [n > 1 for n in self.bx]
        self.ng, self.ndim = m.ng, sum(self.act)
        self.s = [m.ng if a else 0 for a in self.act]
        self.N = [n + 2 * s for n, s in zip(self.bx, self.s)]
        lo, hi = (m.x1min, m.x2min, m.x3min), (m.x1max, m.x2max, m.x3max)
        self.dx = [(b - a) / float(l * n) for a, b, l, n in zip(lo, hi, self.lat, self.bx)]
        b = torch.arange(self.nb, device=dev)
        blk = (b % m.nbx1, (b // m.nbx1) % m.nbx2, b // (m.nbx1 * m.nbx2))
        self.blk = blk
        self.org = [lo[d] + (blk[d] * self.bx[d] - self.s[d]).double() * self.dx[d]
                    for d in range(3)]
        self.I = (slice(None), slice(None)) + tuple(
            slice(self.s[d], self.s[d] + self.bx[d]) for d in (2, 1, 0))
        self.bc = list(m.bc)
        self.heat = bool(self.c["enable_heating"])
        self._met = {}

    def x(self, d, face):
        i = torch.arange(self.N[d] + 1 if face else self.N[d], device=self.dev).double()
        v = self.org[d][:, None] + (i if face else i + 0.5)[None] * self.dx[d]
        shape = [self.nb, 1, 1, 1]
        shape[3 - d] = v.shape[1]
        return v.reshape(shape)

    def gcov(self, x1, x2, x3):
        p, a = self.p, self.p.a
        z = 0.0
        if self.mt == "minkowski":
            one = torch.ones_like(x1)
            return [[(-one if r == 0 else one) if r == c else z * one for c in range(4)]
                    for r in range(4)]
        if self.mt == "cks":
            r2c, a2 = x1 * x1 + x2 * x2 + x3 * x3, a * a
            t = r2c - a2
            r = torch.sqrt(0.5 * (t + torch.sqrt(t * t + 4 * a2 * x3 * x3))).clamp_min(1e-15)
            xi = 2 * r ** 3 / (r ** 4 + a2 * x3 * x3)
            dl = r * r + a2
            l = [1.0, (r * x1 + a * x2) / dl, (r * x2 - a * x1) / dl, x3 / r]
            return [[xi * l[i] * l[j] + ((-1.0 if i == 0 else 1.0) if i == j else 0.0)
                     for j in range(4)] for i in range(4)]
        h, de = p.h, 1e-5

        def theta(y):
            return 0.5 * math.pi * (y + 1) + 0.5 * h * torch.sin(math.pi * (y + 1))

        r, th = torch.exp(x1), theta(x2)
        j1 = (torch.exp(x1 + de) - torch.exp(x1 - de)) / ((x1 + de) - (x1 - de))
        j2 = (theta(x2 + de) - theta(x2 - de)) / ((x2 + de) - (x2 - de))
        cth, sth = torch.cos(th), torch.sin(th)
        s2, r2, a2 = sth * sth, r * r, a * a
        q = [[z * (r * sth)] * 4 for _ in range(4)]
        if self.mt == "mks":
            S = r2 + a2 * cth * cth
            f = 2 * r / S
            q[0][0], q[0][1], q[1][1], q[2][2] = f - 1, f, 1 + f, S
            q[1][0] = f
            q[0][3] = q[3][0] = -2 * a * r * s2 / S
            q[1][3] = q[3][1] = -a * (1 + f) * s2
            q[3][3] = s2 * (S + a2 * s2 * (1 + f))
        else:
            mu = 1 + a2 * cth * cth / r2
            irm = 1 / (r * mu)
            q[0][0], q[1][1], q[2][2] = 2 * irm - 1, mu / (1 - 2 / r + a2 / r2), r2 / mu
            q[0][3] = q[3][0] = -2 * a * s2 * irm
            q[3][3] = r2 * s2 * (1 + a2 / r2 + 2 * a2 * s2 / (r * r2 * mu))
        J = [1.0, j1, j2, 1.0]
        return [[q[i][j] * J[i] * J[j] for j in range(4)] for i in range(4)]

    def metric(self, dire):
        """(gcov, gcon, sqrt|g|, lapse) at centres (0) or at the faces of direction dire."""
        if dire not in self._met:
            g = self.gcov(*[self.x(d, d == dire - 1) for d in range(3)])
            gi, det = _inverse(g)
            self._met[dire] = (g, gi, det.abs().sqrt(), 1 / torch.sqrt(-gi[0][0]))
        return self._met[dire]

    def connection(self):
        x, de = [self.x(d, False) for d in range(3)], 1e-5
        g, gi, _, _ = self.metric(0)
        dg = [[[torch.zeros_like(g[0][0])] * 4 for _ in range(4)]]
        for d in range(3):
            up, dn = list(x), list(x)
            up[d], dn[d] = x[d] + de, x[d] - de
            a, b = self.gcov(*up), self.gcov(*dn)
            dg.append([[(a[i][j] - b[i][j]) / (2 * de) for j in range(4)] for i in range(4)])
        return [[[sum(gi[a][l] * 0.5 * (dg[j][l][k] + dg[k][l][j] - dg[l][j][k])
                      for l in range(4)) for k in range(4)] for j in range(4)] for a in range(4)]

    @staticmethod
    def state(P, met):
        g, gi, _, al = met
        u = P[U1:U1 + 3]
        sq = sum(u[i] * g[i + 1][j + 1] * u[j] for i in range(3) for j in range(3))
        u0 = torch.sqrt(1 + sq) / al
        uc = [u0] + [u[i] - u0 * gi[0][i + 1] * al * al for i in range(3)]
        ul = [sum(g[r][c] * uc[c] for c in range(4)) for r in range(4)]
        b0 = sum(P[B1 + i] * ul[i + 1] for i in range(3))
        bc = [b0] + [(P[B1 + i] + b0 * uc[i + 1]) / u0 for i in range(3)]
        bl = [sum(g[r][c] * bc[c] for c in range(4)) for r in range(4)]
        return uc, ul, bc, bl, sum(bc[i] * bl[i] for i in range(4))

    def flux(self, P, st, sg, d):
        uc, ul, bc, bl, bsq = st
        gam = self.p.adiabatic_index
        et, pt = P[RHO] + gam * P[ENY] + bsq, (gam - 1) * P[ENY] + 0.5 * bsq
        T = [et * uc[d] * ul[m] + (pt if m == d else 0.0) - bc[d] * bl[m] for m in range(4)]
        fr = P[RHO] * uc[d]
        f = [fr, T[0] + fr, T[1], T[2], T[3]]
        f += [bc[i] * uc[d] - bc[d] * uc[i] for i in (1, 2, 3)]
        f += [P[v] * fr for v in range(ENT, len(P))]
        return [v * sg for v in f], T

    def speeds(self, P, st, gi, d):
        uc, bsq, gam = st[0], st[4], self.p.adiabatic_index
        hh = P[RHO] + gam * P[ENY]
        va, cs = bsq / (bsq + hh), gam * (gam - 1) * P[ENY] / hh
        cf = cs + va - cs * va
        cf = torch.where(cf < 0, torch.full_like(cf, 1e-10), cf).clamp_max(1.0)
        n2, t2, nt = uc[d] ** 2, uc[0] ** 2, uc[d] * uc[0]
        A = t2 - (gi[0][0] + t2) * cf
        Bq = 2 * (nt - (gi[0][d] + nt) * cf)
        C = n2 - (gi[d][d] + n2) * cf
        disc = torch.sqrt((Bq * Bq - 4 * A * C).clamp_min(0.0))
        vp, vm = -(disc - Bq) / (2 * A), -(-Bq - disc) / (2 * A)
        return torch.maximum(vp, vm), torch.minimum(vp, vm)

    def recon(self, q):
        """(upper-face value, lower-face value) of the middle cells of a stencil list."""
        if len(q) == 3:
            a, b, c = 2 * (q[1] - q[0]), 0.5 * (q[2] - q[0]), 2 * (q[2] - q[1])
            s = torch.where((a > 0) & (b > 0) & (c > 0), torch.minimum(torch.minimum(a, b), c),
                            torch.zeros_like(a))
            s = torch.where((a < 0) & (b < 0) & (c < 0), torch.maximum(torch.maximum(a, b), c), s)
            return q[1] + 0.5 * s, q[1] - 0.5 * s
        m2, m1, z, p1, p2 = q
        lv, rv = (7 * (z + m1) - (m2 + p1)) / 12, (7 * (z + p1) - (m1 + p2)) / 12
        lv = torch.minimum(torch.maximum(lv, torch.minimum(z, m1)), torch.maximum(z, m1))
        rv = torch.minimum(torch.maximum(rv, torch.minimum(z, p1)), torch.maximum(z, p1))
        c, d = rv - z, lv - z
        flat = c * d >= 0
        r2 = torch.where(c.abs() >= 2 * d.abs(), z - 2 * d, rv)
        l2 = torch.where(d.abs() >= 2 * c.abs(), z - 2 * c, lv)
        return torch.where(flat, z, r2), torch.where(flat, z, l2)

    def fluxes(self, prim):
        """(face fluxes per direction, signal speeds per direction)."""
        mc, out, speed = self.c["limiter"] == "mc", [], []
        hll = self.c["riemann_solver"] == "hll"
        for d in range(1, self.ndim + 1):
            dim, s, n = 5 - d, self.s[d - 1], self.bx[d - 1]
            k = 1 if mc else 2
            q = [prim.narrow(dim, s - 1 + o, n + 2) for o in range(-k, k + 1)]
            up, lo = self.recon(q)
            L, R = up.narrow(dim, 0, n + 1).unbind(1), lo.narrow(dim, 1, n + 1).unbind(1)
            g, gi, sg, al = [self._faces(v, d, s, n) for v in self.metric(d)]
            sL, sR = self.state(L, (g, gi, sg, al)), self.state(R, (g, gi, sg, al))
            (pL, mL), (pR, mR) = self.speeds(L, sL, gi, d), self.speeds(R, sR, gi, d)
            cmax = torch.maximum(pL, pR).clamp_min(0.0)
            cmin = torch.maximum(-mL, -mR).clamp_min(0.0)
            (fL, _), (fR, _) = self.flux(L, sL, sg, d), self.flux(R, sR, sg, d)
            (uL, _), (uR, _) = self.flux(L, sL, sg, 0), self.flux(R, sR, sg, 0)
            ok = (sg > 0) & torch.isfinite(al)
            cms = torch.maximum(cmax, cmin)
            f = torch.zeros_like(prim)
            dst = f.narrow(dim, s, n + 1)
            for v in range(len(fL)):
                if hll:
                    w = (cmax * fL[v] + cmin * fR[v] - cmax * cmin * (uR[v] - uL[v])) / (
                        cmax + cmin + 1e-20)
                else:
                    w = 0.5 * (fL[v] + fR[v] - cms * (uR[v] - uL[v]))
                dst[:, v] = torch.where(ok, w, torch.zeros_like(w))
            if hll and d == 3:  # the transverse range is the interior there
                keep = torch.zeros_like(f)
                sl = list(self.I)
                sl[2] = slice(s, s + n + 1)
                keep[tuple(sl)] = f[tuple(sl)]
                f = keep
            c = torch.zeros_like(prim[:, 0])
            c.narrow(dim - 1, s, n + 1).copy_(torch.where(ok, cms, torch.zeros_like(cms)))
            out.append(f)
            speed.append(c)
        return out, speed

    def _faces(self, v, d, s, n):
        if isinstance(v, list):
            return [self._faces(w, d, s, n) for w in v]
        dim = 4 - d
        return v.narrow(dim, s, n + 1) if v.shape[dim] > 1 else v

    def transport(self, F):
        """Flux-CT: the magnetic face fluxes from the corner fields."""
        a1, a2, a3 = self.act
        sh = lambda t, d, o: torch.roll(t, -o, 4 - d)  # noqa: E731
        f = lambda d, b: F[d - 1][:, B1 + b - 1]  # noqa: E731
        zero = torch.zeros_like(F[0][:, 0])
        e1 = e2 = e3 = zero
        if a2 and a3:
            e1 = 0.25 * (f(2, 3) + sh(f(2, 3), 3, -1) - f(3, 2) - sh(f(3, 2), 2, -1))
        if a3 and a1:
            e2 = 0.25 * (f(3, 1) + sh(f(3, 1), 1, -1) - f(1, 3) - sh(f(1, 3), 3, -1))
        if a1 and a2:
            e3 = 0.25 * (f(1, 2) + sh(f(1, 2), 2, -1) - f(2, 1) - sh(f(2, 1), 1, -1))
        if a1:
            f(1, 1).zero_()
        if a3 and a1:
            f(1, 3).copy_(-0.5 * (e2 + sh(e2, 3, 1)))
            f(3, 1).copy_(0.5 * (e2 + sh(e2, 1, 1)))
        if a1 and a2:
            f(1, 2).copy_(0.5 * (e3 + sh(e3, 2, 1)))
            f(2, 1).copy_(-0.5 * (e3 + sh(e3, 1, 1)))
        if a2 and a3:
            f(2, 3).copy_(0.5 * (e1 + sh(e1, 3, 1)))
            f(3, 2).copy_(-0.5 * (e1 + sh(e1, 2, 1)))
        if a2:
            f(2, 2).zero_()
        if a3:
            f(3, 3).zero_()

    def radius(self):
        x, y, z = [self.x(d, False) for d in range(3)]
        t = x * x + y * y + z * z - self.p.a ** 2
        return torch.sqrt(0.5 * (t + torch.sqrt(t * t + 4 * self.p.a ** 2 * z * z)))

    def fix_primitive(self, prim):
        p, gam, P = self.p, self.p.adiabatic_index, prim.unbind(1)
        met, tiny = self.metric(0), 1e-20
        r = 1.0
        if self.mt == "mks":
            r = torch.exp(self.x(0, False))
        elif self.mt == "cks":
            r = self.radius()
        rr = r.clamp_min(1.0) if torch.is_tensor(r) else torch.ones(1, device=self.dev).double()
        rfl, efl = p.density_floor * rr ** p.density_floor_pow, p.energy_floor * rr ** p.energy_floor_pow
        bsq = self.state(P, met)[4]
        smax = max(p.sigma_max, tiny)
        rfl = torch.maximum(rfl.expand_as(bsq), P[ENY] / smax)
        rfl = torch.where(bsq / P[RHO] > p.sigma_max, bsq / smax, rfl)
        rho, eny = torch.maximum(P[RHO], rfl), torch.maximum(P[ENY], efl)
        g, u = met[0], P[U1:U1 + 3]
        usq = sum(u[i] * g[i + 1][j + 1] * u[j] for i in range(3) for j in range(3))
        umax = p.lorentz_max ** 2 - 1
        f = torch.where(usq > umax, torch.sqrt(umax / usq.clamp_min(tiny)), torch.ones_like(usq))
        u = [v * f for v in u]
        ent = (gam - 1) * eny * rho ** -gam
        out = [rho, eny, *u, *P[B1:B1 + 3], ent]
        if self.heat:
            a, b = rho.clamp_min(tiny), P[RHO].clamp_min(tiny)
            k = torch.where(a != b, P[KEL] * (a / b) ** -gam, P[KEL])
            k = torch.minimum(k, ent).clamp_min(0.0)
            k = torch.minimum(k, ent / (1 + p.ratio_min))
            out.append(torch.maximum(ent / (1 + p.ratio_max), k))
        if self.mt == "cks":
            inside = (r < p.r_excise).expand_as(rho)
            e = p.pexcise / (gam - 1)
            new = [p.dexcise, e, 0.0, 0.0, 0.0, None, None, None,
                   (gam - 1) * e * p.dexcise ** -gam, e]
            out = [v if w is None else _where(inside, w, v) for v, w in zip(out, new)]
        for v, w in enumerate(out):
            prim[:, v] = w

    def _bool_inside(self):
        if self.mt != "cks":
            return None
        return (self.radius() < self.p.r_excise)[self.I[:1] + self.I[2:]]

    def conserved(self, prim, cons):
        met, P = self.metric(0), prim.unbind(1)
        f, _ = self.flux(P, self.state(P, met), met[2], 0)
        for v in range(len(P)):
            if not (self.mixed and B1 <= v < B1 + 3):
                cons[:, v][self.I[1:]] = f[v][self.I[1:]]

    def update(self, F, u0, u1, bdt):
        V = self.dx[0] * self.dx[1] * self.dx[2]
        du = 0.0
        for d in range(self.ndim):
            du = du + (V / self.dx[d]) * (torch.roll(F[d], -1, 4 - d) - F[d])
        u1[self.I] = (u0 - bdt * du / V)[self.I]

    def source(self, prim, cons, bdt):
        if self.mt == "minkowski":
            return
        met, conn, P = self.metric(0), self.connection(), prim.unbind(1)
        st = self.state(P, met)
        T = [self.flux(P, st, met[2], r)[1] for r in range(4)]
        for d in range(4):
            w = sum(T[r][c] * conn[c][d][r] for r in range(4) for c in range(4)) * met[2] * bdt
            cons[:, 1 + d][self.I[1:]] += w[self.I[1:]]

    def exchange(self, a):
        """Block-to-block and periodic ghosts of [block][variable][k][j][i]."""
        bx, s, lat = self.bx, self.s, self.lat
        full = [bx[d] * lat[d] + 2 * s[d] for d in range(3)]
        G = a.new_zeros((a.shape[1], full[2], full[1], full[0]))
        V = torch.zeros(full[2], full[1], full[0], dtype=torch.bool, device=a.device)
        V[tuple(slice(s[d], full[d] - s[d]) for d in (2, 1, 0))] = True

        def at(b, ghosts):
            return tuple(slice(int(self.blk[d][b]) * bx[d] + (0 if ghosts else s[d]),
                               int(self.blk[d][b]) * bx[d] + bx[d] + (2 if ghosts else 1) * s[d])
                         for d in (2, 1, 0))

        for b in range(self.nb):
            G[(slice(None),) + at(b, False)] = a[(b,) + self.I[1:]]
        for d in range(3):
            if s[d] and self.bc[2 * d] == PERIODIC:
                n = full[d] - 2 * s[d]
                for T, dim in ((G, 3 - d), (V, 2 - d)):
                    T.narrow(dim, 0, s[d]).copy_(T.narrow(dim, n, s[d]).clone())
                    T.narrow(dim, n + s[d], s[d]).copy_(T.narrow(dim, s[d], s[d]).clone())
        for b in range(self.nb):
            a[b] = torch.where(V[at(b, True)], G[(slice(None),) + at(b, True)], a[b])

    def boundaries(self, a, signs=True):
        for face in range(6):
            d, outer = face // 2, face % 2
            if not self.act[d] or self.bc[face] == PERIODIC:
                continue
            dim, s, n = 4 - d, self.s[d], self.bx[d]
            own = (self.blk[d] == (self.lat[d] - 1 if outer else 0)).nonzero().flatten()
            x = a[own]
            for q in range(s):
                ghost = s + n + q if outer else s - 1 - q
                edge = s + n - 1 if outer else s
                if self.bc[face] != OUTFLOW:
                    edge = s + n - 1 - q if outer else s + q
                v = x.narrow(dim, edge, 1).clone()
                if self.bc[face] != OUTFLOW and signs:
                    v[:, U1 + d] *= -1
                    v[:, B1 + d] *= -1
                x.narrow(dim, ghost, 1).copy_(v)
            a[own] = x

    # ---- conserved to primitive -------------------------------------------
    def _interior(self, t):
        t = t.expand(self.nb, self.N[2], self.N[1], self.N[0]) if t.dim() == 4 else t
        return t[self.I[:1] + self.I[2:]].reshape(-1)

    def recovery(self, prim, cons, flag):
        met = self.metric(0)
        g = [[self._interior(v) for v in r] for r in met[0]]
        gi = [[self._interior(v) for v in r] for r in met[1]]
        sg, al = self._interior(met[2]), self._interior(met[3])
        C = [self._interior(v) for v in cons.unbind(1)[:9]]
        P = [self._interior(v) for v in prim.unbind(1)[:9]]
        U = [al / sg * v for v in ([C[0], C[1] - C[0]] + C[2:])]
        inside = self._bool_inside()
        live = torch.ones_like(sg, dtype=torch.bool)
        if inside is not None:
            live = ~inside.reshape(-1)
        new = [v.clone() for v in P]
        for k in range(3):
            new[B1 + k] = torch.where(live, C[B1 + k] / sg, P[B1 + k])
        ok = torch.zeros_like(live)
        idx = live.nonzero().flatten()
        take = lambda t: t[idx]  # noqa: E731
        nest = lambda m: [[take(v) for v in r] for r in m]  # noqa: E731
        schemes = ((self._kastaun,) if self.c["recovery"] == "robuster"
                   else (self._newton2d, self._newton_vsq, self._newton_w))
        for scheme in schemes:
            if not idx.numel():
                break
            good, res = scheme([take(v) for v in U], [take(v) for v in P], nest(g), nest(gi))
            w = idx[good]
            for v in range(5):
                new[v][w] = res[v][good]
            ok[w] = True
            idx = idx[~good]
        shape = (self.nb, self.bx[2], self.bx[1], self.bx[0])
        for v in range(9):
            if v != ENT:
                prim[:, v][self.I[:1] + self.I[2:]] = new[v].reshape(shape)
        if self.c["recovery"] != "robuster":
            flag[self.I[:1] + self.I[2:]] = ok.double().reshape(shape)
        return inside

    @staticmethod
    def _harm(U, g, gi):
        B, Q = U[B1:B1 + 3], U[1:5]
        Bl = [sum(g[i + 1][j + 1] * B[j] for j in range(3)) for i in range(3)]
        Qc = [sum(gi[i][j] * Q[j] for j in range(4)) for i in range(4)]
        n0 = -torch.sqrt(-1 / gi[0][0])
        nc = [gi[i][0] * n0 for i in range(4)]
        Bsq, QB = sum(B[i] * Bl[i] for i in range(3)), sum(Q[i + 1] * B[i] for i in range(3))
        Qn = Qc[0] * n0
        Qt = sum(Q[i] * Qc[i] for i in range(4)) + Qn * Qn
        return {"B": B, "Qc": Qc, "nc": nc, "Bsq": Bsq, "QB": QB, "QB2": QB * QB, "Qn": Qn,
                "Qt": Qt, "D": U[0]}

    @staticmethod
    def _velocity(h, G, W):
        return [G / (W + h["Bsq"]) * (h["Qc"][i + 1] + h["nc"][i + 1] * h["Qn"]
                                      + h["QB"] * h["B"][i] / W) for i in range(3)]

    @staticmethod
    def _utsq(P, g):
        u = P[U1:U1 + 3]
        v = sum(u[i] * g[i + 1][j + 1] * u[j] for i in range(3) for j in range(3))
        v = torch.where((v < 0) & (v.abs() < 1e-13), v.abs(), v)
        return v, (v >= 0) & (v <= 1e20)

    @staticmethod
    def _small(W, h):
        return (W ** 3 * (W + 2 * h["Bsq"]) - h["QB2"] * (2 * W + h["Bsq"])
                <= W * W * (h["Qt"] - h["Bsq"] ** 2))

    @staticmethod
    def _newton(step, x, n=30, tol=1e-10):
        """Newton steps with two extra ones after convergence; (x, error, residual)."""
        err, extra = torch.ones_like(x[0]), torch.zeros_like(x[0])
        f, run, began = torch.ones_like(x[0]), torch.ones_like(x[0], dtype=torch.bool), None
        began = torch.zeros_like(run)
        for _ in range(n):
            y, e, r = step(x)
            x = [torch.where(run, b, a) for a, b in zip(x, y)]
            err, f = torch.where(run, e, err), torch.where(run, r, f)
            began = began | (run & (err.abs() <= tol))
            extra = torch.where(run & began, extra + 1, extra)
            run = run & ~(extra > 2)
            if not bool(run.any()):
                break
        return x, err, f

    def _start(self, P, D, ut, h, w0):
        W = w0 * (1 + ut)
        for _ in range(10):
            W = torch.where(self._small(W, h), W * 10, W)
        return W

    def _newton2d(self, U, P, g, gi):
        h, gam = self._harm(U, g, gi), self.p.adiabatic_index
        ut, ok = self._utsq(P, g)
        D, Bs, Q2, Qt, Qn = h["D"], h["Bsq"], h["QB2"], h["Qt"], h["Qn"]
        W = self._start(P, D, ut, h, D / torch.sqrt(1 + ut) + gam * P[ENY])
        vs = ((W * W * Qt + Q2 * (Bs + 2 * W)) / (W * W * (Bs + W) ** 2)).abs()
        vs = torch.where(vs > 1, torch.full_like(vs, 1 - 1e-15), vs)

        def step(x):
            W, v = x
            gt = 1 - v
            s = torch.sqrt(gt)
            p = (gam - 1) * (W * gt - D * s) / gam
            pW, pv = (gam - 1) * gt / gam, (gam - 1) * (0.5 * D / s - W) / gam
            t2, t3, t9 = pv - 0.5 * Bs, Bs + W, 1 / (W * W)
            t4, t16 = t3 * t3, Q2 * t9
            t11 = Qt - v * t4 + Q2 * (Bs + 2 * W) * t9
            t18 = -Qn - 0.5 * Bs * (1 + v) + 0.5 * t16 - W + p
            t24 = t16 / W
            t25 = pW - 1 - t24
            t35 = t25 * t3 + (Bs - 2 * pv) * (Q2 + v * W ** 3) * t9 / W
            a = -(t2 * t11 + t4 * t18) / t3 / t35
            b = -(-t25 * t11 - 2 * (v + t24) * t3 * t18) / t3 / t35
            nW, nv = W + a, v + b
            e = torch.where(nW == 0, a.abs(), (a / nW).abs())
            e = e + torch.where(nv == 0, b.abs(), (b / nv).abs())
            nW = nW.abs()
            nW = torch.where(nW > 1e20, W, nW)
            nv = torch.where(nv > 1, torch.full_like(nv, 1 - 1e-15), nv.clamp_min(0.0))
            return [nW, nv], e, 0.5 * (t11 * t11 + t18 * t18)

        (W, v), err, f = self._newton(step, [W.abs(), vs])
        ok = ok & torch.isfinite(f) & (err.abs() <= 1e-10) & (W > 0) & (W <= 1e20) & (v < 1)
        s = torch.sqrt(1 - v)
        rho, w = D * s, W * (1 - v)
        e = w - (rho + (gam - 1) * (w - rho) / gam)
        return ok & (rho > 0) & (e > 0), [rho, e] + self._velocity(h, 1 / s, W)

    def _newton_vsq(self, U, P, g, gi):
        h, gam, K = self._harm(U, g, gi), self.p.adiabatic_index, P[ENT]
        ut, ok = self._utsq(P, g)
        D, Bs, Q2, Qt = h["D"], h["Bsq"], h["QB2"], h["Qt"]

        def of(v):
            rho = D * torch.sqrt(1 - v)
            p = K * rho ** gam
            return (rho + p / (gam - 1) + p) / (1 - v), p, rho, p / (gam - 1)

        def step(x):
            v, old = x
            W, p, rho, _ = of(v)
            dW = (gam * (2 - gam) * p + (gam - 1) * rho) / (2 * (gam - 1) * (1 - v) ** 2)
            ft = Bs + W
            res = Qt - v * ft * ft + Q2 * (Bs + 2 * W) / (W * W)
            dx = res / (ft * (ft + 2 * dW * (v + Q2 / W ** 3)))
            n = v + dx
            n = torch.where(n >= 1, 0.5 * (v + 1), n)
            n = torch.where(n < -1e-10, 0.5 * v, n).abs()
            W2 = of(n)[0]
            e = torch.where(W2 == 0, (W2 - old).abs(), ((W2 - old) / W2).abs())
            e = e + torch.where(n == 0, (n - v).abs(), ((n - v) / n).abs())
            return [n, W2], e, 0.5 * res * res

        x0 = 1 - 1 / (1 + ut)
        (v, _), err, f = self._newton(step, [x0, torch.zeros_like(x0)])
        ok = ok & torch.isfinite(f) & (err.abs() <= 1e-10) & (v < 1) & (v >= 0)
        W, _, rho, e = of(v)
        return (ok & (rho > 0) & (e > 0),
                [rho, e] + self._velocity(h, 1 / torch.sqrt(1 - v), W))

    def _newton_w(self, U, P, g, gi):
        h, gam, K = self._harm(U, g, gi), self.p.adiabatic_index, P[ENT]
        ut, ok = self._utsq(P, g)
        D, Bs, Q2, Qt = h["D"], h["Bsq"], h["QB2"], h["Qt"]
        rho = D / torch.sqrt(1 + ut)
        p = K * rho ** gam
        W = self._start(P, D, ut, h, rho + p / (gam - 1) + p)
        num = D * D * (1 + gam * K / (gam - 1))

        def step(x):
            W, = x
            D2, r2 = D * D, (num / W) ** 2
            res = (Q2 * D2 * Bs + (2 * Q2 * D2 + ((Qt - Bs * Bs) * D2 + (-2 * D2 * Bs - D2 * W) * W)
                                   * W) * W + (Bs * Bs + (2 * Bs + W) * W) * W * W * r2) / D2 / (W * W)
            jac = -2 * (Q2 * D2 * Bs + (Q2 * D2 + (D2 * Bs + D2 * W) * W * W) * W
                        + (Bs * Bs + Bs * W) * W * W * r2) / D2 / (W * W) / W
            dx = -res / jac
            n = W + dx
            go = torch.ones_like(n, dtype=torch.bool)
            for i in range(10):
                go = go & self._small(n, h)
                n = torch.where(go, n - i * dx / 10, n)
            e = torch.where(n == 0, dx.abs(), (dx / n).abs())
            return [n.abs()], e, 0.5 * res * res

        (W,), err, f = self._newton(step, [W])
        ok = ok & torch.isfinite(f) & torch.isfinite(W) & (err.abs() <= 1e-10)
        v = (W * W * Qt + Q2 * (Bs + 2 * W)) / (W * W * (Bs + W) ** 2)
        ok = ok & (W > 0) & (W <= 1e20) & (v < 1)
        s = torch.sqrt(1 - v)
        rho = D * s
        e = K * rho ** gam / (gam - 1)
        return ok & (rho > 0) & (e > 0), [rho, e] + self._velocity(h, 1 / s, W)

    def _kastaun(self, U, P, g, gi):
        gam, D = self.p.adiabatic_index, U[0]
        gm = [[g[i + 1][j + 1] for j in range(3)] for i in range(3)]
        det = _det3(*[v for r in gm for v in r])
        inv = [[((gm[(j + 1) % 3][(i + 1) % 3] * gm[(j + 2) % 3][(i + 2) % 3]
                  - gm[(j + 1) % 3][(i + 2) % 3] * gm[(j + 2) % 3][(i + 1) % 3]) / det)
                for j in range(3)] for i in range(3)]
        ok = (det > 0) & torch.isfinite(det) & (D > 0) & torch.isfinite(D)
        n0 = -torch.sqrt(-1 / gi[0][0])
        tau = -sum(gi[0][c] * U[1 + c] for c in range(4)) * n0 - D
        S, B = U[2:5], U[B1:B1 + 3]
        Su = [sum(inv[i][j] * S[j] for j in range(3)) for i in range(3)]
        Bl = [sum(gm[i][j] * B[j] for j in range(3)) for i in range(3)]
        b2 = sum(B[i] * Bl[i] for i in range(3)) / D
        r2 = sum(Su[i] * S[i] for i in range(3)) / D / D
        rb = sum(B[i] * S[i] for i in range(3)) / (D * torch.sqrt(D))
        rb2, q = rb * rb, tau / D
        ok = ok & torch.isfinite(tau) & torch.isfinite(b2) & torch.isfinite(r2) & torch.isfinite(rb)

        def parts(mu):
            x = 1 / (1 + mu * b2)
            rbar = x * (r2 * x + mu * (x + 1) * rb2)
            qbar = q - 0.5 * b2 - 0.5 * mu * mu * x * x * (b2 * r2 - rb2)
            return x, rbar, qbar - mu * rbar + 1

        def root(mu):
            x, rbar, eD = parts(mu)
            il = torch.sqrt(1 - (mu * mu * rbar).clamp(0.0, 1 - 1e-14))
            rho = D * il
            eps = (D * eD - rho).clamp_min(1e-300)
            p = (gam - 1) * eps
            nu = torch.maximum((1 + (eps + p) / rho) * il, eD + p / D)
            return mu - 1 / (nu + mu * rbar)

        lo, hi = torch.zeros_like(D), torch.ones_like(D)
        fl, fh = root(lo), root(hi)
        mu = torch.where(fl.abs() <= 1e-10, lo, hi)
        done = ok & torch.isfinite(fl) & torch.isfinite(fh) & (
            (fl.abs() <= 1e-10) | (fh.abs() <= 1e-10))
        run = ok & torch.isfinite(fl) & torch.isfinite(fh) & ~done & (fl * fh <= 0)
        mu, side = torch.where(run, lo, mu), torch.zeros_like(D)
        for _ in range(30):
            new = (fh * lo - fl * hi) / (fh - fl)
            f = root(new)
            old, mu = mu, torch.where(run, new, mu)
            run = run & torch.isfinite(mu) & torch.isfinite(f)
            hit = run & (((mu - old) / (mu + 1e-300)).abs() <= 1e-10)
            done, run = done | hit, run & ~hit
            left = run & (f * fl >= 0)
            right = run & ~left
            wh, wl = 1 - f / fl, 1 - f / fh
            fh = torch.where(left & (side == 1), torch.where(wh > 0, fh * wh, 0.5 * fh), fh)
            fl = torch.where(right & (side == -1), torch.where(wl > 0, fl * wl, 0.5 * fl), fl)
            lo, fl = torch.where(left, mu, lo), torch.where(left, f, fl)
            hi, fh = torch.where(right, mu, hi), torch.where(right, f, fh)
            side = torch.where(left, 1.0, torch.where(right, -1.0, side).double()).double()
        x, rbar, eD = parts(mu)
        v = mu * mu * rbar
        G = 1 / torch.sqrt(1 - v)
        rho = D / G
        eps = D * eD - rho
        ok = done & (v >= 0) & (v < 1) & (rho > 0) & (eps > 0) & torch.isfinite(eps)
        return ok, [rho, eps] + [G * mu * x * (Su[i] / D + rb * mu * B[i] / torch.sqrt(D))
                                 for i in range(3)]

    # ---- after the inversion ----------------------------------------------
    def heating(self, prim, cons):
        if not self.heat:
            return
        p, P, gam = self.p, prim.unbind(1), self.p.adiabatic_index
        ge, gp, name = p.gamma_e, p.gamma_p, self.c["model_name"]
        met = self.metric(0)
        rho, e, bsq = P[RHO], P[ENY], self.state(P, met)[4]
        tot, el = cons[:, ENT] / cons[:, RHO], cons[:, KEL] / cons[:, RHO]
        tp, te = (gp - 1) * e / rho, el * rho ** (ge - 1)
        beta = (2 * rho * tp / bsq)
        beta = torch.where(beta > 1e20, torch.full_like(beta, 1e20), beta)
        fel = torch.full_like(rho, p.fel_constant)
        tr = tp / te
        if name == "howes":
            lt = torch.log(tr) / math.log(10.0)
            low = tr <= 1
            c2, c3 = torch.where(low, 1.6 / tr, 1.2 / tr), torch.where(low, 18 + 5 * lt, 18 + 0 * lt)
            bp = beta ** (2 - 0.2 * lt)
            q = 0.92 * (c2 * c2 + bp) / (c3 * c3 + bp) * torch.exp(-1 / beta) * torch.sqrt(
                1.67262171e-24 / 9.1093826e-28 * tr)
            fel = 1 / (1 + q)
        elif name == "kawazura":
            fel = 1 / (1 + 35 / (1 + (beta / 15) ** -1.4 * torch.exp(-0.1 / tr)))
        elif name == "sharma":
            fel = 1 / (1 + 1 / (0.33 * torch.sqrt(te / tp)))
        rp = rho ** (gam - ge)
        k = el + fel * (ge - 1) / (gam - 1) * rp * (P[ENT] - tot)
        top, low = [tot * rp / (f * (gam - 1) / (gp - 1) + (gam - 1) / (ge - 1))
                    for f in (p.ratio_min, p.ratio_max)]
        k = torch.where(k < top, k, top)
        k = torch.where(low < k, k, low)
        prim[:, KEL][self.I[:1] + self.I[2:]] = k[self.I[:1] + self.I[2:]]

    def fix_recovery(self, prim, flag, inside):
        if self.c["recovery"] == "robuster":
            return
        I = self.I[:1] + self.I[2:]
        bad = torch.zeros_like(flag, dtype=torch.bool)
        bad[I] = flag[I] == 0
        if inside is not None:
            bad[I] &= ~inside.expand_as(bad[I])
        o = 1 if self.act[1] else 0
        at = lambda t, j, i: torch.roll(t, (-j, -i), (-2, -1))  # noqa: E731
        f = lambda j, i: at(flag, j, i) != 0  # noqa: E731
        edge = f(o, 0) & f(0, 1) & f(-o, 0) & f(0, -1)
        diag = f(o, -1) & f(o, 1) & f(-o, 1) & f(-o, -1)
        P0 = prim.clone()
        for v in range(prim.shape[1]):
            q = lambda j, i: at(P0[:, v], j, i)  # noqa: E731
            a = q(o, 0) + q(-o, 0) + q(0, -1) + q(0, 1)
            b = q(o, 1) + q(o, -1) + q(-o, 1) + q(-o, -1)
            w = torch.where(edge, 0.25 * a, torch.where(diag, 0.25 * b, 0.125 * (a + b)))
            prim[:, v] = torch.where(bad, torch.zeros_like(w) if U1 <= v < U1 + 3 else w, prim[:, v])
        flag[bad] = 1.0

    def estimate(self, speed):
        inv = 0.0
        I = self.I[:1] + self.I[2:]
        for d in range(self.ndim):
            m = (self.p.cfl_number * self.dx[d] / speed[d][I]).reshape(self.nb, -1).amin(1)
            inv = inv + 1 / m
        return (1 / inv).amin()

    def stage(self, init, mc0, mc1, flag, beta, dt):
        """mc0, mc1: {prim, cons}; updates both and returns the dt estimate."""
        self.fix_primitive(mc0["prim"])
        self.conserved(mc0["prim"], mc0["cons"])
        F, speed = self.fluxes(mc0["prim"])
        self.transport(F)
        self.update(F, init["cons"], mc1["cons"], beta * dt)
        del F
        self.exchange(mc1["prim"])
        f = flag.unsqueeze(1)
        self.exchange(f)
        self.source(mc1["prim"], mc1["cons"], beta * dt)
        inside = self.recovery(mc1["prim"], mc1["cons"], flag)
        self.heating(mc1["prim"], mc1["cons"])
        self.fix_recovery(mc1["prim"], flag, inside)
        self.boundaries(mc1["prim"])
        self.boundaries(f, signs=False)
        return self.estimate(speed)


def _cycle(c, pin, base, one, flag, dt, factor, tasks=False):
    """The outputs of run() for one job, from its state before it (updated in place)."""
    st = _Stage(pin, c["precision"] == "mixed", base["prim"].device)
    est = st.stage(base, base, one, flag, RK2_BETA[1], dt)
    if tasks:
        return est
    est = st.stage(base, one, base, flag, RK2_BETA[0], dt)
    return torch.minimum(factor * dt, est)


def _state(box):
    if isinstance(box, TableContainer):
        return {f: box.gather(f) for f in ("prim", "cons")}
    return {"prim": box.prim.double(), "cons": box.cons.clone()}


def exact(case, seed):
    c, state = case, prepare(case, seed)
    if "pool" in state:
        pool = state["pool"]
        base, one, flag = _state(pool.base), _state(pool.one), pool.base.flag.clone()
        dt = pool.dt.clone()
        for job, pin in zip(pool.jobs, state["pins"]):
            at = torch.tensor(pool.jobs[job], device=flag.device)
            b, o = ({k: v[at] for k, v in box.items()} for box in (base, one))
            f = flag[at]
            dt[job] = _cycle(c, pin, b, o, f, dt[job].clone(), pool.dt_factor)
            for box, new in ((base, b), (one, o)):
                for k in box:
                    box[k][at] = new[k]
            flag[at] = f
    elif "sim" in state:
        sim = state["sim"]
        base, one, flag = _state(sim.base), _state(sim.one), sim.base.flag.clone()
        dt = _cycle(c, sim.pin, base, one, flag, sim.dt.clone(), sim.dt_factor).reshape(1)
    else:
        base, one = _state(state["base"]), _state(state["one"])
        flag = state["base"].gather("flag")
        est = _cycle(c, state["pin"], base, one, flag, state["dt"], 1.0, tasks=True)
        groups = [0, 1, 2, 5, 8, 9] + ([10] if c["heating"] else [])
        out = {f"{n}_prim": [box["prim"][0, a:b] for a, b in zip(groups, groups[1:])]
               for n, box in (("base", base), ("one", one))}
        out.update(base_cons=[base["cons"][0]], one_cons=[one["cons"][0]], dt=est.reshape(1))
        if c["recovery"] == "chainer":
            out["flag"] = [flag]
        return out
    out = _fields(c, base["prim"])
    out.update(one_prim=one["prim"], base_cons=base["cons"], one_cons=one["cons"], dt=dt)
    if c["recovery"] == "chainer":
        out["flag"] = flag
    return out
