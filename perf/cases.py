"""What a user of this framework has it do, as cases that can be timed and checked.

A case is one particle system (or a batch of them) in motion: the geometries
of this repository (dam breaks, elastic gate, beams, the seeded ensemble) over
the sizes that its configurations name, with a seeded velocity field and, for
the fluids, a seeded displacement of the lattice, as particles have it in the
middle of a run.  A pass goes through the public entry points only:

  steps   GpuSolver.advance(k), then the fields a program saves
  host    sph_step_host(k): the host owns x, v, rho, e (pinned), as the
          reference's time loop does
  rates   nnps() and rates(): the module calls on a state that stays
  batch   GpuBatch.advance(k), then the fields of every system

Passes of `steps`, `host` and `batch` go on from where the last one ended.
Fields of the FP32 pair loops (precision "mixed") are saved in FP32, as the
binary VTK output writes them.  `exact` restates the step in plain torch, in
64 bits, from the formulas of the reference.
"""
import ctypes
import math

import numpy as np
import torch

from mysph_gb300 import cases as geometry
from mysph_gb300 import params as P
from mysph_gb300.solver import GpuBatch, GpuSolver

PRECISION = {"fp64": P.PREC_FP64, "mixed": P.PREC_MIXED, "df64": P.PREC_DF64}
SAVED = ("X", "V", "RHO", "P", "E")


def listed():
    return [
        # the smallest: the reference's cantilever project (505 solid particles), saved every 20 steps
        _case("beam_505_fp64", "steps", "beam", n=505, steps=20),
        # the configuration of 5,000 fluid particles, as it comes and with the lanes that tune_lanes picks for it
        _case("dam2d_5k_fp64", "steps", "dam2d", n=5000, steps=50),
        _case("dam2d_5k_fp64_lanes8", "steps", "dam2d", n=5000, steps=50, lanes=8),
        # the defaults of a project file: normalised summation density, with XSPH
        _case("dam2d_40k_fp64_sumden_xsph", "steps", "dam2d", n=40000, steps=20, sumden=True, xsph=True),
        # a resolution study's larger 2-D run
        _case("dam2d_500k_mixed", "steps", "dam2d", n=500000, steps=50, precision="mixed"),
        # an ordinary 3-D run
        _case("dam3d_26k_fp64", "steps", "dam3d", n=26000, steps=20),
        # the module calls of a fluid-structure case at its configured size (322,000 particles)
        _case("gate_322k_mixed_rates", "rates", "gate", n=322000, precision="mixed"),
        # 3-D in double-float pair loops
        _case("dam3d_214k_df64", "steps", "dam3d", n=214000, steps=20, precision="df64"),
        # the headline workload: the host owns the arrays, one step a call
        _case("dam3d_1700k_fp64_host", "host", "dam3d", n=1690000, steps=1),
        # the same workload in FP32 pair loops
        _case("dam3d_1700k_mixed", "steps", "dam3d", n=1690000, steps=20, precision="mixed"),
        # an ensemble of dam breaks in one batch
        _case("ensemble_64_mixed", "batch", "ensemble", n=2000, n_hi=60000, systems=64, steps=100, precision="mixed"),
        # what a server holds of its solid model: cantilevers of several sizes
        _case("beams_12_mixed", "batch", "beams", n=1000, n_hi=100000, systems=12, steps=50, precision="mixed"),
    ]


def draw(rng):
    kind = rng.choice(["beam", "dam2d", "dam2d", "dam2d", "dam3d", "dam3d", "gate", "host", "ensemble", "beams"])

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    if kind == "beam":
        return _case(None, "steps", "beam", n=size(500, 20000), steps=20)
    if kind == "dam2d":
        n = size(1000, 500000)
        precision = rng.choice(["fp64", "mixed", "df64"])
        more = rng.random() < 0.3 and precision == "fp64"
        lanes = rng.choice([2, 4, 8]) if precision == "fp64" and n < 10000 and rng.random() < 0.5 else 1
        return _case(None, "steps", "dam2d", n=n, steps=20, precision=precision, lanes=lanes, sumden=more, xsph=more)
    if kind == "dam3d":
        return _case(None, "steps", "dam3d", n=size(5000, 800000), steps=10, precision=rng.choice(["fp64", "mixed", "df64"]))
    if kind == "gate":
        return _case(None, "rates", "gate", n=size(10000, 322000), precision=rng.choice(["fp64", "mixed"]))
    if kind == "host":
        return _case(None, "host", rng.choice(["dam2d", "dam3d"]), n=size(2000, 500000), steps=rng.choice([1, 2, 5]))
    count = size(4, 48)
    return _case(None, "batch", kind, n=1000 if kind == "beams" else 2000, n_hi=size(5000, 60000), systems=count,
                 steps=20, precision=rng.choice(["fp64", "mixed"]), pick=rng.randrange(1 << 20))


def _case(name, form, shape, n, steps=1, precision="fp64", lanes=1, sumden=False, xsph=False, n_hi=0, systems=1, pick=7):
    c = dict(name=name, form=form, shape=shape, n=n, steps=steps, precision=precision, lanes=lanes, sumden=sumden,
             xsph=xsph, n_hi=n_hi, systems=systems, pick=pick)
    if name is None:
        del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _geometry(shape, n):
    """The named geometry with about n real particles."""
    if shape == "dam2d":
        return geometry.dam_break_2d(dx=math.sqrt(2.0 / n))
    if shape == "dam3d":
        return geometry.dam_break_3d(dx=(0.108 / n) ** (1.0 / 3.0))
    if shape == "gate":
        return geometry.gate_2d(dx=math.sqrt(0.0805 / n))
    if shape == "beam" and n == 505:
        return geometry.reference_can_beam()
    return geometry.cantilever_2d(dx=math.sqrt(0.004 / n))


def _systems(case):
    """The systems of a case before the seed acts on them."""
    if case["form"] != "batch":
        return [_geometry(case["shape"], case["n"])]
    if case["shape"] == "ensemble":
        return [geometry.ensemble_member(s) for s in
                geometry.ensemble_specs(case["systems"], seed=case["pick"], n_lo=case["n"], n_hi=case["n_hi"])]
    rng = np.random.default_rng(case["pick"])
    sizes = np.exp(rng.uniform(math.log(case["n"]), math.log(case["n_hi"]), case["systems"]))
    return [_geometry("beams", float(k)) for k in sizes]


def _in_motion(c, rng, precision, sumden, xsph):
    """The system with a smooth seeded velocity field, and a displaced lattice where it is a fluid alone."""
    dim, nr = c.dim, c.n_real
    fluid = not np.any(c.type[:nr] > 100)
    x = c.x[:nr]
    size = x.max(0) - x.min(0) + c.meta["dx"]
    speed = (0.03 if fluid else 1e-4) * float(c.c[:nr].max())
    v = np.zeros((nr, dim))
    for _ in range(4):
        k = rng.integers(1, 4, size=dim) * math.pi / size
        v += rng.normal(0.0, 0.5 * speed, size=dim) * np.sin(((x - x.min(0)) * k).sum(1) + rng.uniform(0, 2 * math.pi))[:, None]
    c.v = c.v.copy()
    c.v[:nr] += v
    c.v[c.boundary == 1] = 0.0
    if fluid:
        c.x = c.x.copy()
        c.x[:nr] += rng.uniform(-0.05, 0.05, size=(nr, dim)) * c.meta["dx"]
    c.params = c.params.copy()
    c.params.precision = PRECISION[precision]
    if sumden:
        c.params.flags |= P.F_SUM_DENSITY | P.F_NORM_DENSITY
    if xsph:
        c.params.flags |= P.F_AVER_VELOCITY
    return c


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    return [_in_motion(c, rng, case["precision"], case["sumden"], case["xsph"]) for c in _systems(case)]


def prepare(case, seed):
    systems = _inputs(case, seed)
    state = dict(case=case)
    if case["form"] == "batch":
        b = GpuBatch(systems[0].params, len(systems), sum(c.n_real for c in systems), sum(c.n_wall for c in systems) + 1)
        state["ids"] = [b.add(c) for c in systems]
        state["batch"] = b
        return state
    c = systems[0]
    state["solver"] = s = GpuSolver(c)
    if case["lanes"] > 1:
        s.set_option(P.OPT_LANES, case["lanes"])
    if case["form"] == "host":
        nr = c.n_real
        state["host"] = [torch.from_numpy(np.ascontiguousarray(a[:nr])).pin_memory() for a in (c.x, c.v, c.rho, c.e)]
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _saved(a, precision):
    return a.astype(np.float32) if precision == "mixed" else a


def run(state):
    case = state["case"]
    form, precision, steps = case["form"], case["precision"], case["steps"]
    if form == "batch":
        b = state["batch"]
        b.advance(steps)
        return {f: np.concatenate([_saved(b.field(k, f), precision).ravel() for k in state["ids"]]) for f in ("X", "V", "RHO")}
    s = state["solver"]
    if form == "host":
        dp = ctypes.POINTER(ctypes.c_double)
        s._call("sph_step_host", steps, *[ctypes.cast(a.data_ptr(), dp) for a in state["host"]], None)
        return dict(zip("xvre", state["host"]))
    if form == "rates":
        s.nnps()
        return [_saved(a, precision) for a in s.rates()]
    s.advance(steps)
    return {f: _saved(s.field(f), precision) for f in SAVED}


def work(case):
    """Bytes: each step reads and writes the evolving state of every real particle (x, v, rho, e, with a solid's stress)
    and reads what stays (mass, h, c, type; the walls' x, mass, rho, p, h). Operations: those of the formulas, per pair."""
    systems = _systems(case)
    steps = 1 if case["form"] == "rates" else case["steps"]
    total = flops = 0
    for c in systems:
        solid = bool(np.any(c.type[: c.n_real] > 100))
        state = 2 * c.dim + 2 + (c.dim * c.dim if solid else 0)
        total += c.n_real * (16 * state + 28) + c.n_wall * 8 * (c.dim + 4)
        pairs = {2: 20, 3: 56}[c.dim]
        flops += c.n_real * pairs * {2: 100, 3: 150}[c.dim] + c.n_real * (pairs * 25 if case["sumden"] else 0)
    return {"bytes": total * steps, "flops": flops * steps}


# ---------------------------------------------------------------------------
# the same pass in plain torch, in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    m = _Step(_inputs(case, seed))
    nr, dim = m.nr, m.dim
    if case["form"] == "rates":
        m.search()
        m.rates()
        return [m.a, m.drho, m.de]
    for _ in range(case["steps"]):
        m.step()
    if case["form"] == "host":
        return dict(x=m.x[:nr], v=m.v[:nr], r=m.rho[:nr], e=m.e[:nr])
    if case["form"] == "batch":
        # the fields of system k: its real particles, then its walls
        order = torch.argsort(m.sys, stable=True)
        return {"X": m.x[order].reshape(-1), "V": m.v[order].reshape(-1), "RHO": m.rho[order]}
    return {"X": m.x, "V": m.v, "RHO": m.rho, "P": m.p, "E": m.e}


class _Step:
    """Several independent systems, their real particles first and all walls after them, stepped by the leap-frog of the reference."""

    CHUNK = 1 << 27   # candidate pairs looked at in one go

    def __init__(self, systems):
        dev = self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        f8 = torch.float64
        prm = self.prm = systems[0].params
        self.dim = d = int(prm.dim)
        self.nr = sum(c.n_real for c in systems)

        def both(get, dtype=f8):
            parts = [get(c)[: c.n_real] for c in systems] + [get(c)[c.n_real:] for c in systems]
            return torch.from_numpy(np.concatenate(parts)).to(dev, dtype)

        def per(get, dtype=f8):
            return torch.tensor([get(c) for c in systems], dtype=dtype, device=dev)

        self.sys = both(lambda c: np.full(c.n, systems.index(c)), torch.int64)
        self.x, self.v = both(lambda c: c.x), both(lambda c: c.v)
        self.m, self.rho, self.e = both(lambda c: c.mass), both(lambda c: c.rho), both(lambda c: c.e)
        self.c, self.h, self.p = both(lambda c: c.c), both(lambda c: c.h), both(lambda c: c.p)
        self.type, self.fixed = both(lambda c: c.type, torch.int64), both(lambda c: c.boundary, torch.int64)[: self.nr] == 1
        self.S = both(lambda c: np.zeros((c.n, d * d)) if c.shear is None else c.shear).view(-1, d, d).transpose(1, 2)
        sr = self.sys[: self.nr]
        self.dt = per(lambda c: c.params.dt)[sr]
        self.r0, self.delta, self.dp = (per(g)[self.sys] for g in (lambda c: c.params.wall_r0, lambda c: c.params.contact_delta, lambda c: c.params.as_dp))
        # the material of each particle: one row per system and |type|
        self.rho0, self.B, self.gamma, self.K, self.eta = (torch.zeros(len(self.m), dtype=f8, device=dev) for _ in range(5))
        self.linear = torch.zeros(len(self.m), dtype=torch.bool, device=dev)
        for k, c in enumerate(systems):
            for q in range(c.params.n_materials):
                w = c.params.materials[q]
                at = (self.sys == k) & (self.type.abs() == w.type)
                self.rho0[at], self.gamma[at], self.K[at], self.eta[at] = w.rho0, w.gamma, w.K, w.eta
                self.B[at] = w.c0 * w.c0 * w.rho0 / w.gamma if w.gamma else 0.0
                self.linear[at] = w.eos == P.EOS_LINEAR
        self.solid = self.type.abs() > 100
        self.p = self.eos()                              # walls keep theirs; a real particle's is set in rates()
        self.divx = torch.zeros(self.nr, dtype=f8, device=dev)
        self.n_step = 0
        # a grid of cells of 2h per system
        self.cell = per(lambda c: 2.0 * float(c.h.max()) * (1 + 1e-9))
        self.lo = torch.stack([torch.tensor(c.x.min(0), dtype=f8) for c in systems]).to(dev) - 6 * self.cell[:, None]
        hi = torch.stack([torch.tensor(c.x.max(0), dtype=f8) for c in systems]).to(dev) + 6 * self.cell[:, None]
        self.nc = ((hi - self.lo) / self.cell[:, None]).long() + 1
        self.base = torch.cumsum(self.nc.prod(1), 0) - self.nc.prod(1)

    def flag(self, f):
        return bool(self.prm.flags & f)

    def eos(self):
        return torch.where(self.linear, self.K / self.rho0 * (self.rho - self.rho0),
                           self.B * ((self.rho / self.rho0) ** self.gamma - 1.0))

    def kernel(self, r, h):
        """Cubic spline: W(r, h) and dW/dx = g dx."""
        f = 15.0 / (7.0 * math.pi * h * h) if self.dim == 2 else 3.0 / (2.0 * math.pi * h ** 3)
        q = r / h
        inner, t = q < 1.0, 2.0 - q
        w = torch.where(inner, f * (2.0 / 3.0 - q * q + 0.5 * q ** 3), f / 6.0 * t ** 3)
        g = torch.where(inner, f * (-2.0 + 1.5 * q) / (h * h), -0.5 * f * t * t / (h * r.clamp_min(1e-300)))
        return w, g

    def search(self):
        """Targets i and neighbours j (r < 2 h_i), by target."""
        cell = ((self.x - self.lo[self.sys]) / self.cell[self.sys][:, None]).long()
        cell = torch.maximum(torch.minimum(cell, self.nc[self.sys] - 1), torch.zeros_like(cell))
        nc, base = self.nc[self.sys], self.base[self.sys]

        def key(c):
            k = c[:, 1] if self.dim == 2 else c[:, 2] * nc[: len(c), 1] + c[:, 1]
            return base[: len(c)] + k * nc[: len(c), 0] + c[:, 0]

        keys, order = torch.sort(key(cell), stable=True)
        rows = [(y, z) for z in ((0,) if self.dim == 2 else (-1, 0, 1)) for y in (-1, 0, 1)]
        starts, counts = [], []
        for y, z in rows:
            c = cell[: self.nr].clone()
            c[:, 1] += y
            if self.dim == 3:
                c[:, 2] += z
            k = key(c)
            starts.append(torch.searchsorted(keys, k - 1))
            counts.append(torch.searchsorted(keys, k + 1, right=True) - starts[-1])
        starts, counts = torch.stack(starts, 1), torch.stack(counts, 1)
        per = counts.sum(1)
        ends = torch.cumsum(per, 0)
        got_i, got_j, first = [], [], 0
        while first < self.nr:
            done = int(ends[first - 1]) if first else 0
            last = max(first + 1, int(torch.searchsorted(ends, done + self.CHUNK, right=True)))
            cnt = counts[first:last].reshape(-1)
            i = torch.repeat_interleave(torch.arange(first, last, device=self.dev), per[first:last])
            off = torch.cumsum(cnt, 0) - cnt
            j = order[torch.arange(len(i), device=self.dev) + torch.repeat_interleave(starts[first:last].reshape(-1) - off, cnt)]
            r = (self.x[i] - self.x[j]).square_().sum(1).sqrt_()
            near = (r < 2.0 * self.h[i]) & (i != j)
            got_i.append(i[near])
            got_j.append(j[near])
            first = last
        self.i, self.j = torch.cat(got_i), torch.cat(got_j)
        self.lengths = torch.bincount(self.i, minlength=self.nr)

    def chunks(self):
        """The pairs in pieces that hold whole targets."""
        ends = torch.cumsum(self.lengths, 0)
        first = done = 0
        while first < self.nr:
            last = max(first + 1, int(torch.searchsorted(ends, done + self.CHUNK // 4, right=True)))
            stop = int(ends[last - 1])
            i, j = self.i[done:stop], self.j[done:stop]
            dx = self.x[i] - self.x[j]
            r = dx.square().sum(1).sqrt()
            yield first, last, i, j, dx, r
            first, done = last, stop

    def total(self, first, last, term):
        return torch.segment_reduce(term.contiguous(), "sum", lengths=self.lengths[first:last], axis=0, initial=0.0, unsafe=True)

    def density(self):
        rho = torch.empty(self.nr, dtype=torch.float64, device=self.dev)
        for a, b, i, j, dx, r in self.chunks():
            w, _ = self.kernel(r, self.h[i])
            w0, _ = self.kernel(torch.zeros_like(self.h[a:b]), self.h[a:b])
            s = self.m[a:b] * w0 + self.total(a, b, self.m[j] * w)
            shep = self.V[a:b] * w0 + self.total(a, b, self.V[j] * w)
            norm = (self.divx[a:b] < 1.5) & self.flag(P.F_NORM_DENSITY)
            rho[a:b] = torch.where(norm, s / shep, s)
        self.rho[: self.nr] = rho
        self.V = self.m / self.rho

    def rates(self):
        nr, d, prm = self.nr, self.dim, self.prm
        f8 = dict(dtype=torch.float64, device=self.dev)
        self.V = self.m / self.rho
        if self.flag(P.F_SUM_DENSITY):
            self.density()
        # velocity gradient, continuity, strain; EOS and stresses
        G, sdx, aver = torch.empty(nr, d, d, **f8), torch.empty(nr, **f8), torch.zeros(nr, d, **f8)
        for a, b, i, j, dx, r in self.chunks():
            w, g = self.kernel(r, self.h[i])
            vg = self.V[j] * g
            dv = self.v[j] - self.v[i]
            G[a:b] = self.total(a, b, ((vg[:, None] * dv)[:, :, None] * dx[:, None, :]).flatten(1)).view(-1, d, d)
            sdx[a:b] = self.total(a, b, vg * r * r)
            if self.flag(P.F_AVER_VELOCITY):
                aver[a:b] = self.total(a, b, (2.0 * prm.xsph_eps * self.m[j] / (self.rho[i] + self.rho[j]) * w)[:, None] * dv)
        aver[self.fixed] = 0.0
        self.aver, self.divx = aver, -sdx
        divv = G.diagonal(dim1=1, dim2=2).sum(1)
        rho = self.rho[:nr]
        self.drho = torch.zeros_like(rho) if self.flag(P.F_SUM_DENSITY) else -rho * divv
        p = self.eos()
        self.p = torch.cat([p[:nr], self.p[nr:]])
        eye = torch.eye(d, **f8)
        solid = self.solid[:nr][:, None, None]
        edot = torch.where(solid, 0.5 * (G + G.transpose(1, 2)), 2.0 * G - (2.0 / 3.0) * divv[:, None, None] * eye)
        eta, S, pr = self.eta[:nr], self.S[:nr], self.p[:nr][:, None, None]
        dev = edot - edot.diagonal(dim1=1, dim2=2).sum(1)[:, None, None] / 3.0 * eye
        rot = 0.5 * (G - G.transpose(1, 2))
        tds = torch.where(self.solid[:nr], (S * dev).sum((1, 2)), 0.5 * eta * edot.square().sum((1, 2))) / rho
        self.dS = torch.where(solid, 2.0 * eta[:, None, None] * dev + S @ rot.transpose(1, 2) + rot @ S.transpose(1, 2), torch.zeros_like(S))
        sig = torch.zeros(len(self.m), d, d, **f8)
        sig[:nr] = torch.where(solid, S - pr * eye, torch.zeros_like(S)) / rho[:, None, None] ** 2
        T = -(self.p / self.rho ** 2)[:, None, None] * eye
        visc = eta[:, None, None] * edot
        if self.flag(P.F_FSI_FLUID_VISCOUS):
            visc = torch.where(solid, torch.zeros_like(visc), visc)
        T[:nr] += visc / rho[:, None, None] ** 2
        R = None
        if self.flag(P.F_ARTI_STRESS) and d == 2:
            R = torch.zeros(len(self.m), d, d, **f8)
            R[:nr] = torch.where(self.type[:nr][:, None, None] >= 100, self.stress_r(S - pr * eye, rho), R[:nr])
        # momentum and energy
        Pm = self.p / self.rho ** 2
        self.a, self.de = torch.empty(nr, d, **f8), torch.empty(nr, **f8)
        for a, b, i, j, dx, r in self.chunks():
            w, g = self.kernel(r, self.h[i])
            w_ = (self.m[j] * g)[:, None] * dx
            dv = self.v[i] - self.v[j]
            si = self.solid[i][:, None]
            pair = torch.where(si[:, :, None], sig[i] + sig[j], T[i] + T[j])
            acc = (pair * w_[:, None, :]).sum(2)
            dvw = (dv * w_).sum(1)
            en = 0.5 * (Pm[i] + Pm[j]) * dvw
            xv = (dx * dv).sum(1)
            if self.flag(P.F_ARTI_VISC):
                so = self.type[i] > 100
                al = prm.av_alpha + (prm.av_alpha_solid - prm.av_alpha) * so.double()
                be = prm.av_beta + (prm.av_beta_solid - prm.av_beta) * so.double()
                hij, rij, cij = (0.5 * (q[i] + q[j]) for q in (self.h, self.rho, self.c))
                phi = hij * xv / (r * r + (prm.av_psi * hij) ** 2)
                PI = torch.where(xv < 0, (be * phi - al * cij) * phi / rij, torch.zeros_like(phi))
                acc -= PI[:, None] * w_
                en += 0.5 * PI * dvw
            f = self.external(i, j, r)
            if f is not None:
                acc += f[:, None] * dx
            if R is not None:
                wd, _ = self.kernel(self.dp[i], self.h[i])
                F = torch.where(self.type[j] >= 100, (w / wd) ** prm.as_n, torch.zeros_like(w))
                acc += ((R[i] + R[j]) * (F[:, None] * w_)[:, None, :]).sum(2)
            self.a[a:b] = self.total(a, b, acc)
            self.de[a:b] = self.total(a, b, en)
        self.de += tds
        if self.flag(P.F_GRAVITY):
            heavy = ~(self.type[:nr] > 100) if self.flag(P.F_GRAVITY_SKIP_SOLIDS) else torch.ones_like(self.fixed)
            self.a[:, d - 1] += prm.gravity * heavy.double()
        self.a[self.fixed] = 0.0

    def external(self, i, j, r):
        """Wall repulsion and fluid-solid contact: the factor of dx."""
        prm, ti, tj = self.prm, self.type[i], self.type[j]
        if not self.flag(P.F_EXT_FORCE | P.F_DUMMY | P.F_GRAVITY):
            return None
        r = r.clamp_min(1e-300)
        t = self.r0[i] / r
        zero = torch.zeros_like(r)
        f = torch.where((ti > 0) & (tj < 0) & (r < self.r0[i]), prm.wall_fs * (t ** prm.wall_p1 - t ** prm.wall_p2) / (r * r), zero)
        contact = (tj > 0) & (ti > 0) & (ti != tj) & ~((ti > 100) & (tj > 100)) & ((ti > 100) | (tj > 100))
        eta = r / 0.75 / (0.5 * (self.h[i] + self.h[j]))
        chi = 1.0 - r / self.delta[i]
        chi = torch.where((chi < 0) | (chi > 1), zero, chi)
        fc = torch.where(eta <= 2.0 / 3.0, torch.full_like(eta, 2.0 / 3.0), torch.where(eta <= 1.0, 2.0 * eta - 1.5 * eta * eta, 0.5 * (2.0 - eta) ** 2))
        fc = torch.where((eta <= 0) | (eta >= 2), zero, fc)
        return f + torch.where(contact, P.f32(0.01) * self.c[i] ** 2 * chi * fc / (r * r), zero)

    def stress_r(self, s, rho):
        """The artificial-stress tensor of a 2-D solid with stress s."""
        aux = s[:, 0, 0] - s[:, 1, 1]
        th = 0.5 * torch.atan((s[:, 0, 1] + s[:, 1, 0]) / torch.where(aux == 0, torch.ones_like(aux), aux))
        th = torch.where(aux == 0, torch.full_like(aux, 0.5 * math.pi), th)
        cs, sn = th.cos(), th.sin()
        p0 = cs * cs * s[:, 0, 0] + sn * sn * s[:, 1, 1] + 2 * sn * cs * s[:, 0, 1]
        p1 = sn * sn * s[:, 0, 0] + cs * cs * s[:, 1, 1] - 2 * sn * cs * s[:, 0, 1]
        t0, t1 = (torch.where(q > 0, -self.prm.as_eps * q / rho ** 2, torch.zeros_like(q)) for q in (p0, p1))
        off = sn * cs * (t0 - t1)
        return torch.stack([cs * cs * t0 + sn * sn * t1, off, off, sn * sn * t0 + cs * cs * t1], 1).view(-1, 2, 2)

    def step(self):
        nr, dt, summed = self.nr, self.dt, self.flag(P.F_SUM_DENSITY)
        dt1, dt2 = dt[:, None], dt[:, None, None]
        solid = self.solid[:nr][:, None, None]
        e0, rho0, v0, S0 = (q[:nr].clone() for q in (self.e, self.rho, self.v, self.S))
        if self.n_step:
            self.e[:nr] = (e0 + dt / 2 * self.de).clamp_min(0.0)
            if not summed:
                self.rho[:nr] = rho0 + dt / 2 * self.drho
            self.v[:nr] = v0 + dt1 / 2 * self.a
            self.S[:nr] = torch.where(solid, S0 + dt2 / 2 * self.dS, S0)
        self.search()
        self.rates()
        full = 1.0 if self.n_step else 0.5
        self.e[:nr] = (e0 + full * dt * self.de).clamp_min(0.0)
        if not summed:
            self.rho[:nr] = rho0 + full * dt * self.drho
        self.v[:nr] = v0 + full * dt1 * self.a + self.aver
        self.x[:nr] += dt1 * self.v[:nr]
        self.S[:nr] = torch.where(solid, S0 + full * dt2 * self.dS, S0)
        self.n_step += 1
