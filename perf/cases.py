"""The calls whose speed and results are followed: time steps of the 2-D solver in both precisions
from the smallest grid to the largest, a step driven routine by routine, a batch of ragged
cases, the discrete adjoint, and the 3-D LES step.

A pass is what a program that owns the flow arrays does: the state goes from page-locked
host memory into the context, the steps run, the state comes back.  Grids, time steps and
Poisson settings are those of the benchmark, the tests and the reference's defaults.  The
number of Poisson sweeps of a step is fixed by the cap (the tolerance lies below what the
line iteration reaches in that many sweeps), except in the smallest case, which keeps the
reference's own tolerance.
"""
import math

import numpy as np
import torch

from fvm_gb300 import batch as fbatch
from fvm_gb300 import capi, capi3d
from fvm_gb300.grid import o_grid, o_grid_3d

R = 0.5   # cylinder radius
STATE2 = ("U", "V", "P", "T", "NLX", "NLY", "ADV")
NEVER = 1e-14   # a Poisson tolerance that the capped iteration does not reach


def listed():
    return [
        # the smallest call: the reference's own Poisson settings on the smoke test's grid
        dict(name="step2d 32x24 fp64 default", kind="step2d", theta=32, r=24, prec="fp64", re=100.0, dt=0.005,
             sweeps=20, tol=1e-4, every=1, refine=4, steps=1, skew=0.0, rot=0.0, thermal=True, driver="step"),
        # a driver that calls the reference's routines one by one, skewed grid, rotating wall, odd radial count
        dict(name="points2d 200x131 fp64 skew", kind="step2d", theta=200, r=131, prec="fp64", re=150.0, dt=0.002,
             sweeps=24, tol=NEVER, every=2, refine=4, steps=1, skew=0.2, rot=0.3, thermal=True, driver="points"),
        # the laminar shedding case, Re 100, in FP64
        dict(name="step2d 128x96 fp64", kind="step2d", theta=128, r=96, prec="fp64", re=100.0, dt=0.005,
             sweeps=512, tol=NEVER, every=8, refine=16, steps=1, skew=0.0, rot=0.0, thermal=False, driver="step"),
        # the same grid in mixed precision, a stretch of a run
        dict(name="step2d 128x96 mixed", kind="step2d", theta=128, r=96, prec="mixed", re=100.0, dt=0.005,
             sweeps=512, tol=NEVER, every=8, refine=16, steps=4, skew=0.0, rot=0.0, thermal=False, driver="step"),
        # the benchmark's workload: Re 200 with temperature, 2048 sweeps a step, mixed and FP64
        dict(name="step2d 512x384 mixed", kind="step2d", theta=512, r=384, prec="mixed", re=200.0, dt=0.002,
             sweeps=2048, tol=NEVER, every=8, refine=32, steps=2, skew=0.0, rot=0.0, thermal=True, driver="step"),
        dict(name="step2d 512x384 fp64", kind="step2d", theta=512, r=384, prec="fp64", re=200.0, dt=0.002,
             sweeps=2048, tol=NEVER, every=8, refine=32, steps=1, skew=0.0, rot=0.0, thermal=True, driver="step"),
        # the sweep over 64 ragged cases
        dict(name="batch2d 64 ragged mixed", kind="batch2d", cases=64, theta_max=256, r_max=192, prec="mixed",
             dt=0.004, sweeps=512, every=8, refine=32, steps=2),
        # reverse mode: one transposed step, and the drag gradient over a checkpointed window
        dict(name="adjoint vjp 128x96 mixed", kind="vjp2d", theta=128, r=96, prec="mixed", re=100.0, dt=0.005,
             sweeps=512, every=8, refine=16),
        dict(name="adjoint window 128x96 fp64", kind="window2d", theta=128, r=96, prec="fp64", re=100.0, dt=0.005,
             sweeps=128, every=8, refine=16, window=6, ckpt=3),
        # 3-D LES: a small grid with the reference's sweep count, the profiled grid in FP64, the benchmark's in mixed
        dict(name="les3d 64x48x16 mixed", kind="les3d", theta=64, r=48, z=16, prec="mixed", dr1=0.01, dt=0.002,
             sweeps=20, refine=4, every=2, steps=2, les=True),
        dict(name="les3d 192x160x32 fp64", kind="les3d", theta=192, r=160, z=32, prec="fp64", dr1=0.001, dt=0.002,
             sweeps=64, refine=8, every=4, steps=1, les=True),
        dict(name="les3d 256x192x48 mixed", kind="les3d", theta=256, r=192, z=48, prec="mixed", dr1=0.001, dt=0.002,
             sweeps=200, refine=8, every=8, steps=2, les=True),
    ]


def _log(rng, a, b):
    return math.exp(rng.uniform(math.log(a), math.log(b)))


def draw(rng):
    kind = rng.choice(["step2d", "step2d", "step2d", "batch2d", "vjp2d", "window2d", "les3d", "les3d"])
    prec = rng.choice(["fp64", "mixed", "mixed"])
    theta = 4 * round(_log(rng, 32, 512) / 4)
    r = round(_log(rng, 24, 384))
    refine = rng.choice([4, 8, 16, 32])
    if kind == "step2d":
        sweeps = refine * max(1, round(_log(rng, 16, 1024) / refine))
        return dict(kind=kind, theta=theta, r=r, prec=prec, re=_log(rng, 60, 300), dt=rng.choice([0.002, 0.004, 0.005]),
                    sweeps=sweeps, tol=NEVER, every=rng.choice([2, 4, 8]) if sweeps % 8 == 0 else 2, refine=refine,
                    steps=rng.choice([1, 1, 2, 4]), skew=rng.choice([0.0, 0.0, 0.2]), rot=rng.choice([0.0, 0.3]),
                    thermal=rng.random() < 0.6, driver=rng.choice(["step", "step", "points"]))
    if kind == "batch2d":
        return dict(kind=kind, cases=round(_log(rng, 2, 64)), theta_max=rng.choice([96, 160, 256]),
                    r_max=rng.randint(64, 192), prec=prec, dt=0.004, sweeps=refine * max(1, 128 // refine), every=8,
                    refine=refine, steps=rng.choice([1, 2]))
    theta, r = 4 * round(_log(rng, 32, 256) / 4), round(_log(rng, 24, 192))
    if kind == "vjp2d":
        return dict(kind=kind, theta=theta, r=r, prec=prec, re=_log(rng, 60, 300), dt=0.005,
                    sweeps=refine * max(1, round(_log(rng, 32, 512) / refine)), every=8, refine=refine)
    if kind == "window2d":
        return dict(kind=kind, theta=theta, r=r, prec=prec, re=_log(rng, 60, 300), dt=0.005, sweeps=64, every=8,
                    refine=refine, window=rng.randint(2, 6), ckpt=rng.randint(1, 4))
    z = 2 * rng.randint(4, 20)
    if prec == "fp64":
        theta, r, z = min(theta, 160), min(r, 128), min(z, 24)
    return dict(kind=kind, theta=theta, r=r, z=z, prec=prec, dr1=rng.choice([0.002, 0.005]), dt=0.001,
                sweeps=refine * max(1, round(_log(rng, 20, 160) / refine)), refine=refine, every=4,
                steps=rng.choice([1, 2]), les=rng.random() < 0.8)


# ---------------------------------------------------------------------------------
# Inputs: a cylinder flow with a wall layer and seeded large-scale disturbances
# ---------------------------------------------------------------------------------
def _flow(r, th, rng, z=None, lz=1.0):
    """u, v, w, p, t at polar points (r, th) of a solenoidal flow past the cylinder: the potential
    flow's stream function times a wall-layer factor, seeded modes of a second stream
    function that vanishes with its gradient at the wall (modulated along the span in 3-D)
    and a spanwise velocity of the same form.  Pressure: Bernoulli's of the outer flow."""
    s, d = r - R, 0.15
    g = torch.tanh(s / d)
    h = (r - R * R / r) * g
    hp = (1.0 + R * R / (r * r)) * g + (r - R * R / r) * (1.0 - g * g) / d
    ur, ut = h / r * torch.cos(th), -hp * torch.sin(th)
    w = torch.zeros_like(ur)
    q, qp = s * s * torch.exp(-s), (2.0 * s - s * s) * torch.exp(-s)
    for m in range(1, 7):
        a, ph = 0.06 * rng.standard_normal() / m, rng.uniform(0.0, 2.0 * math.pi)
        b, pz = 0.05 * rng.standard_normal() / m, rng.uniform(0.0, 2.0 * math.pi)
        cz = 1.0 if z is None else 1.0 + 0.5 * torch.cos(2.0 * math.pi * (1 + m % 3) * z / lz + pz)
        ur = ur - a * m * q / r * torch.sin(m * th + ph) * cz
        ut = ut - a * qp * torch.cos(m * th + ph) * cz
        w = w + b * q * torch.cos(m * th + pz)
    u, v = ur * torch.cos(th) - ut * torch.sin(th), ur * torch.sin(th) + ut * torch.cos(th)
    k = (R / r) ** 2
    p = 0.5 * (2.0 * k * torch.cos(2.0 * th) - k * k)
    t = torch.exp(-s / 0.2) * (1.0 + 0.1 * torch.cos(th + rng.uniform(0.0, 6.28)))
    return u, v, w, p, t


def _state2(g, rot, seed):
    """The seven state arrays (rows j = 0..NJ, columns i = 0..NI) with the ghost cells of the boundary conditions."""
    rng = np.random.default_rng(seed)
    xc = 0.25 * (g.xg[2:, 2:] + g.xg[1:-1, 2:] + g.xg[2:, 1:-1] + g.xg[1:-1, 1:-1])
    yc = 0.25 * (g.yg[2:, 2:] + g.yg[1:-1, 2:] + g.yg[2:, 1:-1] + g.yg[1:-1, 1:-1])
    x, y = torch.from_numpy(xc), torch.from_numpy(yc)
    u, v, _, p, t = _flow(torch.hypot(x, y), torch.atan2(y, x), rng)
    th = torch.atan2(y[:, 0], x[:, 0])
    wall = {"U": -rot * torch.sin(th), "V": rot * torch.cos(th), "T": torch.ones_like(th)}
    far = {"U": 1.0, "V": 0.0, "T": 0.0}
    out = {nm: torch.zeros((g.nj + 1, g.ni + 1), dtype=torch.float64) for nm in STATE2}
    for nm, f in (("U", u), ("V", v), ("P", p), ("T", t)):
        a = out[nm]
        a[1:-1, 1:-1] = f
        if nm == "P":
            a[1:-1, 0] = f[:, 0]
            a[1:-1, -1] = 3.0 * f[:, -1] - 3.0 * f[:, -2] + f[:, -3]
        else:
            a[1:-1, 0] = 2.0 * wall[nm] - f[:, 0]
            a[1:-1, -1] = 2.0 * far[nm] - f[:, -1]
        a[0], a[-1] = a[-2], a[1]
    return out


def _pinned(arrays):
    return {nm: a.cpu().contiguous().pin_memory() for nm, a in arrays.items()}


def _blank(arrays):
    return {nm: torch.empty(a.shape, dtype=torch.float64).pin_memory() for nm, a in arrays.items()}


def _ptrs(arrays):
    return [a.data_ptr() for a in arrays.values()]


def _params2(c, ni, nj, re=None):
    return capi.default_params(ni=ni, nj=nj, re=c["re"] if re is None else re, dt=c["dt"], nswpp=c["sweeps"],
                               resimax=c.get("tol", NEVER), res_every=c["every"], refine_sweeps=c["refine"],
                               vel_rot=c.get("rot", 0.0), thermal=int(c.get("thermal", False)),
                               precision=capi.MIXED if c["prec"] == "mixed" else capi.FP64)


def _context2(c, g, re=None):
    ctx = capi.Context(_params2(c, g.ni, g.nj, re))
    ctx.set_grid(g.xg, g.yg)
    ctx.init()
    return ctx


def _specs(c):
    return fbatch.sweep_cases(c["cases"], seed=0, dt=c["dt"], theta=(64, c["theta_max"], 16), radial=(48, c["r_max"]))


def _state3(c, g, seed):
    rng = np.random.default_rng(seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x2 = 0.25 * (g.xg[1, 2:, 2:] + g.xg[1, 1:-1, 2:] + g.xg[1, 2:, 1:-1] + g.xg[1, 1:-1, 1:-1])
    y2 = 0.25 * (g.yg[1, 2:, 2:] + g.yg[1, 1:-1, 2:] + g.yg[1, 2:, 1:-1] + g.yg[1, 1:-1, 1:-1])
    x, y = torch.from_numpy(x2).to(dev)[None], torch.from_numpy(y2).to(dev)[None]
    z = (torch.arange(g.nk - 1, device=dev, dtype=torch.float64) + 0.5).reshape(-1, 1, 1) * (g.lz / (g.nk - 1))
    f = _flow(torch.hypot(x, y), torch.atan2(y, x), rng, z, g.lz)
    out = {}
    for nm, a, wall, far in zip(("U", "V", "W", "P", "T"), f, (0.0, 0.0, 0.0, None, 1.0), (1.0, 0.0, 0.0, None, 0.0)):
        a = a.expand(g.nk - 1, g.nj - 1, g.ni - 1)
        full = torch.zeros((g.nk + 1, g.nj + 1, g.ni + 1), dtype=torch.float64, device=dev)
        full[1:-1, 1:-1, 1:-1] = a
        full[1:-1, 1:-1, 0] = a[..., 0] if wall is None else 2.0 * wall - a[..., 0]
        full[1:-1, 1:-1, -1] = 3.0 * a[..., -1] - 3.0 * a[..., -2] + a[..., -3] if far is None else 2.0 * far - a[..., -1]
        full[:, 0], full[:, -1] = full[:, -2].clone(), full[:, 1].clone()
        full[0], full[-1] = full[-2].clone(), full[1].clone()
        out[nm] = full
    for nm in ("NLX", "NLY", "NLZ", "ADV"):
        out[nm] = torch.zeros_like(out["U"])
    return out


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "les3d":
        g = o_grid_3d(c["theta"], c["r"], c["z"], dr1=c["dr1"])
        p = capi3d.default_params(ni=g.ni, nj=g.nj, nk=g.nk, dt=c["dt"], nswpp=c["sweeps"], resimax=NEVER,
                                  refine_sweeps=c["refine"], res_every=c["every"], use_les=int(c["les"]), ref_a=g.lz,
                                  precision=capi.MIXED if c["prec"] == "mixed" else capi.FP64, poisson_host_loop=0)
        ctx = capi3d.Context3(p)
        ctx.set_grid(g)
        src = _pinned(_state3(c, g, seed))
        return dict(kind=kind, ctx=ctx, src=src, dst=_blank(src), steps=c["steps"])
    if kind == "batch2d":
        specs = _specs(c)
        grids = [o_grid(s.n_theta, s.n_r) for s in specs]
        b = capi.Batch([_params2(c, g.ni, g.nj, s.re) for g, s in zip(grids, specs)])
        for ctx, g in zip(b.cases, grids):
            ctx.set_grid(g.xg, g.yg)
            ctx.init()
        src = [_pinned(_state2(g, 0.0, seed * 1000 + k)) for k, g in enumerate(grids)]
        return dict(kind=kind, ctx=b, src=src, dst=[_blank(s) for s in src], steps=c["steps"])
    g = o_grid(c["theta"], c["r"], skew=c.get("skew", 0.0))
    ctx = _context2(c, g)
    src = _pinned(_state2(g, c.get("rot", 0.0), seed))
    st = dict(kind=kind, ctx=ctx, src=src, dst=_blank(src), steps=c.get("steps", 1), driver=c.get("driver", "step"),
              thermal=bool(c.get("thermal", False)))
    if kind == "vjp2d":
        rng = np.random.default_rng(seed + 77)
        ctx.upload_ptrs(_ptrs(src))
        st["lam"] = {nm: rng.standard_normal((g.nj + 1, g.ni + 1)) for nm in ("U", "V", "P", "NLX", "NLY")}
    if kind == "window2d":
        st.update(window=c["window"], ckpt=c["ckpt"])
    return st


# the record's entries that are results of the flow (not the clock or the iteration's residual norm)
def _record(rec):
    return [rec[k] for k in ("cfl", "cpb", "cd", "cl", "cd_p", "cd_v", "cl_p", "cl_v", "nu")]


def _points(ctx, thermal):
    """One time step through the entry points that stand for the reference's subroutines, in its order."""
    ctx.begin_step()
    ctx.contra_vel()
    for f in (capi.FIELD_U, capi.FIELD_V) + ((capi.FIELD_T,) if thermal else ()):
        ctx.nl(f)
        ctx.dif(f)
    ctx.p_source()
    ctx.iter_u()
    ctx.iter_v()
    ctx.remove_grad()
    ctx.iter_p()
    ctx.correct()
    if thermal:
        ctx.iter_t()
    return ctx.calccoef()


def run(state):
    ctx, kind = state["ctx"], state["kind"]
    if kind == "batch2d":
        for c, s in zip(ctx.cases, state["src"]):
            c.upload_ptrs(_ptrs(s))
        rec = ctx.step(state["steps"])[-1]
        for c, d in zip(ctx.cases, state["dst"]):
            c.download_ptrs(_ptrs(d))
        out = {nm: torch.cat([d[nm].reshape(-1) for d in state["dst"]]) for nm in STATE2}
        out["record"] = np.array([_record(r) for r in rec])
        out["sweeps"] = np.array([r["sweeps"] for r in rec])
        return out
    if kind == "vjp2d":
        lam, omega, blow = ctx.adjoint_vjp(state["lam"])
        return dict(lam, omega=omega, blow=blow)
    ctx.upload_ptrs(_ptrs(state["src"]))
    if kind == "window2d":
        J, omega, blow = ctx.adjoint_drag_grad(state["window"], state["ckpt"])
        ctx.download_ptrs(_ptrs(state["dst"]))
        return dict(state["dst"], J=J, omega=omega, blow=blow)
    if kind == "step2d" and state["driver"] == "points":
        for _ in range(state["steps"]):
            rec = _points(ctx, state["thermal"])
    else:
        rec = ctx.step(state["steps"])
    ctx.download_ptrs(_ptrs(state["dst"]))
    return dict(state["dst"], record=np.array(_record(rec)), sweeps=rec["sweeps"])


def work(case):
    """Bytes: the state and the node coordinates read once, the state written once (the adjoint: its
    adjoint state in and out besides, and the window's checkpoints once each way).
    Operations per cell: 9 a Poisson sweep (two couplings, two recurrences of the line
    solve), 25 a residual, and those of the explicit terms and predictor lines of a step."""
    c, kind = case, case["kind"]
    if kind == "les3d":
        n = c["theta"] * c["r"] * c["z"]
        per = 13 * c["sweeps"] + 50 * c["sweeps"] / max(c["refine"], c["every"]) + 700 + (900 if c["les"] else 0)
        return dict(bytes=8.0 * n * (9 + 3 + 9), flops=n * per * c["steps"])
    if kind == "batch2d":
        n = sum(s.cells for s in _specs(c))
    else:
        n = c["theta"] * c["r"]
    per = 9 * c["sweeps"] + 25 * c["sweeps"] / max(c["refine"], c["every"]) + 250 + (90 if c.get("thermal") else 0)
    if kind == "vjp2d":
        return dict(bytes=8.0 * n * (2 + 2 + 5 + 5), flops=n * per)
    if kind == "window2d":
        k = -(-c["window"] // c["ckpt"])
        return dict(bytes=8.0 * n * (7 + 2 + 7 + 14 * k), flops=3.0 * n * per * c["window"])
    return dict(bytes=8.0 * n * (7 + 2 + 7), flops=n * per * c.get("steps", 1))


# ---------------------------------------------------------------------------------
# The 2-D time step restated in 64 bits with plain torch (arrays [j, i], ghosts included)
# ---------------------------------------------------------------------------------
class _Plain2:
    """The same discrete step and sweep order (odd lines, then even ones, periodic wrap; cyclic lines
    around the cylinder), every line system solved with its dense inverse."""

    def __init__(self, c, g, state, re):
        self.c, self.dt, self.re, self.pe = c, c["dt"], re, re * 0.71
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.f = {nm: a.to(self.dev).clone() for nm, a in state.items()}
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)   # noqa: E731
        xg, yg = t(g.xg), t(g.yg)

        def centres(q):
            a = torch.zeros_like(q)
            a[1:-1, 1:-1] = 0.25 * (q[2:, 2:] + q[1:-1, 2:] + q[2:, 1:-1] + q[1:-1, 1:-1])
            a[1:-1, 0] = (q[2:, 1] + q[1:-1, 1]) - a[1:-1, 1]
            a[1:-1, -1] = (q[2:, -1] + q[1:-1, -1]) - a[1:-1, -2]
            return self.wrap(a)

        X, Y = centres(xg), centres(yg)

        def d_xi(a):
            b = torch.zeros_like(a)
            b[:, 1:-1] = 0.5 * (a[:, 2:] - a[:, :-2])
            b[:, 0] = 0.5 * (-3.0 * a[:, 0] + 4.0 * a[:, 1] - a[:, 2])
            b[:, -1] = 0.5 * (3.0 * a[:, -1] - 4.0 * a[:, -2] + a[:, -3])
            return b

        def d_eta(a):
            b = torch.zeros_like(a)
            b[1:-1] = 0.5 * (a[2:] - a[:-2])
            return self.wrap(b)

        xx, xe, yx, ye = d_xi(X), d_eta(X), d_xi(Y), d_eta(Y)
        J = self.J = xx * ye - yx * xe
        self.xix, self.xiy, self.etx, self.ety = ye / J, -xe / J, -yx / J, xx / J
        q11, q22 = self.xix ** 2 + self.xiy ** 2, self.etx ** 2 + self.ety ** 2
        self.jq12 = J * (self.xix * self.etx + self.xiy * self.ety)
        self.D = self.faces(J * q11, J * q22)
        th = torch.remainder(torch.atan2(Y, X), 2.0 * math.pi)
        rot, tw = c.get("rot", 0.0), th[1:-1, 0]
        self.wall = {"U": -rot * torch.sin(tw), "V": rot * torch.cos(tw), "T": torch.ones_like(tw)}
        tf = th[1:-1, -1]
        self.inflow = (tf >= 0.5 * math.pi) & (tf <= 1.5 * math.pi)
        self.systems = {}
        for nm, rek in (("mom", self.re), ("heat", self.pe)) if c.get("thermal") else (("mom", self.re),):
            for k, (m1, m2) in enumerate(((self.xix, self.etx), (self.xiy, self.ety))):
                E, W, N, S = self.faces(J * m1 * m1, J * m2 * m2)
                P = 2.0 * rek * self.inner(J) / self.dt + E + W + N + S
                raw = (W[:, 0].clone(), E[:, -1].clone())
                P[:, 0] += W[:, 0]
                P[:, -1] += E[:, -1]
                W[:, 0] = 0.0
                E[:, -1] = 0.0
                inv = self.inverse(P, W, E, False) if k == 0 else self.inverse(P.T, S.T, N.T, True)
                self.systems[nm, k] = (E, W, N, S, raw, inv)
        E, W, N, S = (-a for a in self.D)
        P = E + W + N + S
        P[:, 0] -= W[:, 0]
        W[:, 0] = 0.0
        E[:, -1] = 0.0
        self.poisson = (E, W, N, S, P, self.inverse(P, W, E, False))

    @staticmethod
    def wrap(a):
        a[0], a[-1] = a[-2], a[1]
        return a

    @staticmethod
    def inner(a, dj=0, di=0):
        nj, ni = a.shape
        return a[1 + dj:nj - 1 + dj, 1 + di:ni - 1 + di]

    def faces(self, a, b):
        n = self.inner
        return (0.5 * (n(a) + n(a, 0, 1)), 0.5 * (n(a) + n(a, 0, -1)), 0.5 * (n(b) + n(b, 1)), 0.5 * (n(b) + n(b, -1)))

    def inverse(self, P, lo, hi, cyclic):
        """Inverses of the systems P x - lo x(-1) - hi x(+1), a line per row."""
        n = P.shape[1]
        A = torch.zeros((P.shape[0], n, n), dtype=torch.float64, device=self.dev)
        k = torch.arange(n, device=self.dev)
        A[:, k, k] = P
        A[:, k[1:], k[:-1]] = -lo[:, 1:]
        A[:, k[:-1], k[1:]] = -hi[:, :-1]
        if cyclic:
            A[:, 0, -1] = -lo[:, 0]
            A[:, -1, 0] = -hi[:, -1]
        return torch.linalg.inv(A)

    @staticmethod
    def zebra(inv, rhs, put):
        for c in (0, 1):
            put(c, torch.bmm(inv[c::2], rhs(c)[:, :, None])[:, :, 0])

    def cross(self, K, f):
        n = self.inner
        return 0.25 * (n(K, 0, 1) * (n(f, 1, 1) - n(f, -1, 1)) - n(K, 0, -1) * (n(f, 1, -1) - n(f, -1, -1))
                       + n(K, 1) * (n(f, 1, 1) - n(f, 1, -1)) - n(K, -1) * (n(f, -1, 1) - n(f, -1, -1)))

    def shifted(self, f):
        """The cross term as the whole-array sum pairs it: cell (i, j) takes that of (i-1, j-1)."""
        d, q = self.cross(self.jq12, f), torch.zeros_like(self.D[0])
        q[1:, 1:] = d[:-1, :-1]
        return q

    def ghosts(self, nm, far):
        a = self.f[nm]
        a[1:-1, 0] = 2.0 * self.wall[nm] - a[1:-1, 1]
        a[1:-1, -1] = 2.0 * far[nm] - a[1:-1, -2]
        self.wrap(a)

    def p_ghosts(self):
        a = self.f["P"]
        a[1:-1, 0] = a[1:-1, 1]
        a[1:-1, -1] = 3.0 * a[1:-1, -2] - 3.0 * a[1:-1, -3] + a[1:-1, -4]
        self.wrap(a)

    def fluxes(self):
        u, v, J = self.f["U"], self.f["V"], self.J
        E, W, N, S = self.faces(J * (self.xix * u + self.xiy * v), J * (self.etx * u + self.ety * v))
        W[:, 0] = 0.0
        return E, W, N, S

    def grad_p(self):
        n, P, J = self.inner, self.f["P"], self.J
        return [-0.5 * (n(J * a * P, 0, 1) - n(J * a * P, 0, -1) + n(J * b * P, 1) - n(J * b * P, -1))
                for a, b in ((self.xix, self.etx), (self.xiy, self.ety))]

    def predictor(self, nm, old, nl, nm1, dif, src, far):
        n, rek = self.inner, self.pe if nm == "T" else self.re
        a, kind = self.f[nm], "heat" if nm == "T" else "mom"
        JD = 2.0 * rek * n(self.J) / self.dt
        su = JD * n(old) - 3.0 * rek * nl + rek * nm1 + dif + self.cross(self.J * self.xix * self.etx, a)
        if src is not None:
            su = su + 2.0 * rek * src
        for k in (0, 1):
            E, W, N, S, raw, inv = self.systems[kind, k]
            if k == 1:
                x = self.f["V"] if nm == "T" else a   # the reference builds this term of T from V
                su = JD * n(a) + self.cross(self.J * self.xiy * self.ety, x)
            su[:, 0] += 2.0 * raw[0] * self.wall[nm]
            su[:, -1] += 2.0 * raw[1] * far[nm]
            self.ghosts(nm, far)
            inside = n(a)

            def put(c, x, k=k):
                if k == 0:
                    inside[c::2] = x
                else:
                    inside[:, c::2] = x.T

            def rhs(c, k=k):
                if k == 0:
                    s = inside
                    return (N * torch.roll(s, -1, 0) + S * torch.roll(s, 1, 0) + su)[c::2]
                return (E * n(a, 0, 1) + W * n(a, 0, -1) + su)[:, c::2].T

            self.zebra(inv, rhs, put)

    def solve_p(self, div):
        c, P, n = self.c, self.f["P"], self.inner
        E, W, N, S, AP, inv = self.poisson
        mixed = c["prec"] == "mixed"
        per = c["refine"] if mixed else max(2, c["every"] + c["every"] % 2)
        cap = -(-c["sweeps"] // per) * per
        tol = c.get("tol", NEVER)

        def sweep(x, su):
            self.zebra(inv, lambda k: (N * torch.roll(x, -1, 0) + S * torch.roll(x, 1, 0) + su)[k::2],
                       lambda k, v: x[k::2].copy_(v))

        def resid(su):
            p = n(P)
            r = E * n(P, 0, 1) + W * n(P, 0, -1) + N * torch.roll(p, -1, 0) + S * torch.roll(p, 1, 0) + su - AP * p
            return r, float(r.abs().sum() / (AP * p).abs().sum())

        it = 0
        while True:
            if mixed:
                r, s = resid(div - self.shifted(P))
                if it and not (s > tol and it < cap):
                    break
                x = torch.zeros_like(r)
                for _ in range(per):
                    sweep(x, r)
                n(P).add_(x)
                self.p_ghosts()
                it += per
            else:
                for _ in range(per):
                    su = div - self.shifted(P)
                    self.p_ghosts()
                    sweep(n(P), su)
                it += per
                if not (resid(su)[1] > tol and it < cap):
                    break
        self.p_ghosts()
        return it

    def step(self):
        n, f, dt = self.inner, self.f, self.dt
        fields = ("U", "V", "T") if self.c.get("thermal") else ("U", "V")
        hist = {"U": "NLX", "V": "NLY", "T": "ADV"}
        old = {nm: f[nm].clone() for nm in ("U", "V", "T")}
        far = {}
        a = 0.5 * (self.xix[1:-1, -1] + self.xix[1:-1, -2])
        b = 0.125 * (self.etx[1:-1, -1] + self.etx[1:-1, -2])
        for nm, inflow in (("U", 1.0), ("V", 0.0), ("T", 0.0)):
            q = old[nm]
            dq = q[2:, -1] + q[2:, -2] - q[:-2, -1] - q[:-2, -2]
            out = 0.5 * (q[1:-1, -1] + q[1:-1, -2]) - dt * (a * (q[1:-1, -1] - q[1:-1, -2]) + b * dq)
            far[nm] = torch.where(self.inflow, torch.full_like(out, inflow), out)
        E, W, N, S = self.fluxes()
        DE, DW, DN, DS = self.D
        su = dict(zip(("U", "V"), self.grad_p()))
        terms = {}
        for nm in fields:
            q, c = old[nm], n(old[nm])
            e, w, no, so = n(q, 0, 1), n(q, 0, -1), n(q, 1), n(q, -1)
            nl = 0.5 * (E * (c + e) - W * (c + w) + N * (c + no) - S * (c + so))
            dif = DE * (e - c) + DW * (w - c) + DN * (no - c) + DS * (so - c) + self.shifted(q)
            terms[nm] = (nl, n(f[hist[nm]]).clone(), dif)
            n(f[hist[nm]]).copy_(nl)
        for nm in ("U", "V"):
            self.predictor(nm, old[nm], *terms[nm], su[nm], far)
        for nm in ("U", "V"):
            n(f[nm]).sub_(dt * su[nm] / n(self.J))
            self.ghosts(nm, far)
        E, W, N, S = self.fluxes()
        self.sweeps = self.solve_p((E - W + N - S) / dt)
        for nm, s in zip(("U", "V"), self.grad_p()):
            n(f[nm]).add_(dt * s / n(self.J))
            self.ghosts(nm, far)
        if "T" in fields:
            self.predictor("T", old["T"], *terms["T"], None, far)
            self.ghosts("T", far)


def exact(case, seed):
    """The 2-D steps' states.  The adjoint and the LES step have no counterpart that plain torch
    gives: their outputs are held to the start's."""
    c, kind = case, case["kind"]
    if kind == "batch2d":
        outs = []
        for k, s in enumerate(_specs(c)):
            g = o_grid(s.n_theta, s.n_r)
            m = _Plain2(c, g, _state2(g, 0.0, seed * 1000 + k), s.re)
            for _ in range(c["steps"]):
                m.step()
            outs.append({nm: m.f[nm].cpu().reshape(-1) for nm in STATE2})
            del m
        return dict({nm: torch.cat([o[nm] for o in outs]) for nm in STATE2}, record=None, sweeps=None)
    if kind != "step2d":
        return None
    g = o_grid(c["theta"], c["r"], skew=c["skew"])
    m = _Plain2(c, g, _state2(g, c["rot"], seed), c["re"])
    for _ in range(c["steps"]):
        m.step()
    return dict({nm: m.f[nm].cpu() for nm in STATE2}, record=None, sweeps=m.sweeps)
