"""Performance cases of the channel-flow library, through its public entry points.

Every case is a dict of plain values.  ``kind`` says what a pass does:

    steps        Channel.step(n), the statistics and the solution copied out: the time
                 loop of a run between two outputs (float64 or mixed precision, RK2 or
                 RK3, plain or variant walls, with or without the diagnostics series)
    restart      init_sol_v from a host field, a few steps, statistics, solution out:
                 a restart segment on ordinary (pageable) host arrays
    sweep        Ensemble.step(n) over a stratified parameter sweep of uneven grids
    closure_run  steps of a coarse run with the learned subgrid closure attached
    train        one epoch of the closure's training
    infer        closure outputs for host inputs
    sample       a training set from a DNS snapshot: filter, sample, normalise, read back
    post         fluctuation field and Q-criterion of a stored state

``exact`` restates each of them in plain torch in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from compchan3dmpi_b200 import Channel, ChanParams
from compchan3dmpi_b200.closure import Closure, attach
from compchan3dmpi_b200.ensemble import Ensemble
from compchan3dmpi_b200.wallbc import WallBC, spanwise_stripes

DEV = "cuda"
F64 = torch.float64
CFL = 0.5
PLANES = (5, 10, 16)          # x-planes of the diagnostics series


# ---------------------------------------------------------------- the cases
def _steps(name, n1, n2, n3, steps, rk=3, mixed=False, mesh="tanh", wall="plain", istat=10, diag=0, kind="steps"):
    c = dict(kind=kind, n1=n1, n2=n2, n3=n3, steps=steps, rk=rk, mixed=mixed, mesh=mesh, wall=wall, istat=istat,
             diag=diag)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: one step of a toy grid, watched step by step
        _steps("toy_step_24x14x19", 24, 14, 19, 1, rk=2, mesh="cosine", istat=1),
        # the reference's own configuration: RK2, cosine mesh, 64 x 48 x 65
        _steps("reference_64x48x65", 64, 48, 65, 50, rk=2, mesh="cosine"),
        # a ragged grid with slip stripes on the bottom wall and the diagnostics series
        _steps("stripes_101x75x83", 101, 75, 83, 40, wall="slip", diag=10),
        # the production DNS grid, plain FP64 and mixed precision
        _steps("dns_256x192x193", 256, 192, 193, 50),
        _steps("dns_mixed_256x192x193", 256, 192, 193, 50, mixed=True),
        # restart from a host field and write the solution back
        _steps("restart_160x128x129", 160, 128, 129, 10, kind="restart"),
        # the stratified sweep: 16 uneven mixed-precision cases stepped as one ensemble
        dict(name="sweep_16_mixed", kind="sweep", members=16, lo=64, hi=160, steps=20, mixed=True),
        # a coarse run with the learned closure
        dict(name="closure_run_64x64x65", kind="closure_run", n1=64, n2=64, n3=65, steps=20, hold=True),
        # closure training: one epoch of a million samples at the usual batch
        dict(name="train_1M", kind="train", n=1 << 20, batch=65536),
        # closure outputs for a host batch, an odd number of rows
        dict(name="infer_50001", kind="infer", n=50001),
        # training data from a DNS snapshot, the filter and strides of the experiment
        dict(name="sample_256x192x97", kind="sample", n1=256, n2=192, n3=97, sx=4, sy=3, sz=3, width=4),
        # post-processing of a stored state
        dict(name="post_128x96x97", kind="post", n1=128, n2=96, n3=97),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "restart", "sweep", "closure_run", "train", "infer", "sample",
                       "post"])
    if kind == "steps":
        grid = (_log(rng, 20, 256), _log(rng, 12, 192), _log(rng, 17, 193))
        return _steps(None, *grid, _log(rng, 1, 50), rk=rng.choice([2, 3, 3]), mixed=rng.random() < 0.4,
                      mesh=rng.choice(["cosine", "tanh"]), wall=rng.choice(["plain", "plain", "slip", "hot"]),
                      istat=rng.choice([1, 5, 10]), diag=rng.choice([0, 0, 10]))
    if kind == "restart":
        return _steps(None, _log(rng, 32, 180), _log(rng, 24, 140), _log(rng, 25, 140), _log(rng, 2, 20), kind=kind)
    if kind == "sweep":
        lo = _log(rng, 40, 80)
        return dict(kind=kind, members=rng.randint(2, 12), lo=lo, hi=lo + _log(rng, 8, 80), steps=10 * rng.randint(1, 2),
                    mixed=rng.random() < 0.7)
    if kind == "closure_run":
        return dict(kind=kind, n1=_log(rng, 32, 96), n2=_log(rng, 32, 96), n3=_log(rng, 33, 97),
                    steps=_log(rng, 2, 20), hold=rng.random() < 0.7)
    if kind == "train":
        batch = 128 * _log(rng, 8, 512)
        return dict(kind=kind, n=batch * rng.randint(1, 16) + rng.randint(0, 999), batch=batch)
    if kind == "infer":
        return dict(kind=kind, n=_log(rng, 1, 200000))
    if kind == "sample":
        return dict(kind=kind, n1=_log(rng, 48, 256), n2=_log(rng, 40, 192), n3=_log(rng, 33, 129),
                    sx=rng.choice([1, 2, 4]), sy=rng.choice([2, 3]), sz=rng.choice([2, 3]),
                    width=rng.choice([2, 4]))
    return dict(kind=kind, n1=_log(rng, 32, 160), n2=_log(rng, 32, 128), n3=_log(rng, 33, 129))


# ------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _mesh(n3, kind):
    xi = 2.0 * np.arange(n3) / (n3 - 1)
    if kind == "cosine":
        x3, jac = 1.0 - np.cos(0.5 * xi * math.pi), 0.5 * math.pi * np.sin(0.5 * xi * math.pi)
        inv = np.zeros(n3)
        inv[1:] = 1.0 / jac[1:]
        return x3, jac, inv
    beta = 2.2
    th = np.tanh(beta * (xi - 1.0))
    x3, jac = 1.0 + th / math.tanh(beta), beta * (1.0 - th * th) / math.tanh(beta)
    x3[0], x3[-1] = 0.0, 2.0
    return x3, jac, 1.0 / jac


def _full(a):
    """Stored points from the unique periodic ones (the last two axes)."""
    a = torch.cat([a[..., -1:], a, a[..., :1]], -1)
    return torch.cat([a[..., -1:, :], a, a[..., :1, :]], -2)


def _start(p, x3, seed, amp=0.15):
    """Laminar profile, smooth perturbations and grid-scale noise between walls at p.Tw: var[7, nP3, nP2, nP1]."""
    n1, n2, n3 = p.nP
    g = _gen(seed)
    z = torch.tensor(x3, device=DEV, dtype=F64)[:, None, None]
    y = (torch.arange(n2 - 2, device=DEV, dtype=F64) * (2 * math.pi / (n2 - 2)))[None, :, None]
    x = (torch.arange(n1 - 2, device=DEV, dtype=F64) * (2 * math.pi / (n1 - 2)))[None, None, :]
    lam = 1.5 * (1.0 - (z - 1.0) ** 2)
    lam[0] = lam[-1] = 0.0
    vel = []
    for c in range(3):
        ph = torch.rand(6, generator=g, device=DEV, dtype=F64) * 2 * math.pi
        d = sum(torch.cos(kx * x + ky * y + ph[n]) for n, (kx, ky) in
                enumerate([(1, 1), (2, 1), (1, 2), (3, 1), (2, 3), (4, 2)]))
        noise = torch.rand((n3, n2 - 2, n1 - 2), generator=g, device=DEV, dtype=F64) * 2 - 1
        vel.append((lam if c == 0 else 0) + amp * lam * (0.25 * d + 0.3 * noise))
    Tb, Tt = p.Tw
    T = Tb + (Tt - Tb) * 0.5 * z + 0.3 * lam * (2.0 - lam) / 1.5 - 0.2 * (vel[0] - lam)
    rho = 1.0 / T
    u, v, w = vel
    E = T + 0.5 * p.ggM * (u * u + v * v + w * w)
    return _full(torch.stack([rho, u, v, w, E, T, rho * T / (p.gama * p.Mac ** 2)]))


def _with_dt(p, var, jac, cfl=CFL):
    k = slice(1, -1)
    rho, u, v, w, T = (var[m][k, k, k] for m in (0, 1, 2, 3, 5))
    dz = torch.tensor(p.dXi * jac[1:-1], device=DEV, dtype=F64)[:, None, None]
    c = T.sqrt() / p.Mac
    lam = (u.abs() + c) / p.dx + (v.abs() + c) / p.dy + (w.abs() + c) / dz
    nu = T.pow(0.7) / (rho * p.Re)
    lam += 2 * max(4 / 3, p.gama / p.Pr) * nu * (1 / p.dx ** 2 + 1 / p.dy ** 2 + 1 / dz ** 2)
    return p.with_(dt=float(cfl / lam.max()))


def _flow(case, seed):
    """(params, mesh, var on the device, wall variant) of a single-grid case."""
    hot = case.get("wall") == "hot"
    # the Reynolds number a grid resolves: 3000 from 64 x 48 x 65 on, lower on coarser grids
    res = min(1.0, case["n1"] / 64, case["n2"] / 48, case["n3"] / 65)
    p = ChanParams(nP=(case["n1"], case["n2"], case["n3"]), Re=3000.0 * res * res, Pr=0.72 if case.get("rk", 3) == 3 else 0.71,
                   rk_scheme=case.get("rk", 3), mixed=case.get("mixed", False), istat=case.get("istat", 10),
                   Tw=(1.0, 1.2) if hot else (1.0, 1.0))
    mesh = _mesh(case["n3"], case.get("mesh", "tanh"))
    var = _start(p, mesh[0], seed)
    return _with_dt(p, var, mesh[1]), mesh, var


def _members(case, seed):
    """The members of a stratified sweep: uneven grids, (Ma, Re, Ri, dT) in turn."""
    out = []
    n, lo, hi = case["members"], case["lo"], case["hi"]
    for c in range(n):
        f = [((c * s) % n) / max(n - 1, 1) for s in (1, 5, 3)]
        grid = (lo + round(f[0] * (hi - lo)), lo + round(f[1] * 0.67 * (hi - lo)), lo + 1 + round(f[2] * 0.67 * (hi - lo)))
        dT, Ri = (0.0, 0.2)[c % 2], (0.0, 0.1, 0.5)[c % 3]
        p = ChanParams(nP=grid, Re=(2000.0, 3000.0, 4000.0)[(c // 2) % 3], Mac=(0.5, 1.5)[(c // 3) % 2], Pr=0.72,
                       rk_scheme=3, istat=10, Tw=(1.0 - dT / 2, 1.0 + dT / 2), mixed=case["mixed"])
        mesh = _mesh(grid[2], "tanh")
        var = _start(p, mesh[0], seed * 64 + c)
        out.append((_with_dt(p, var, mesh[1]), mesh, var, Ri))
    return out


def _features(n, seed):
    """Training samples: inputs with the spread of velocity gradients, targets that depend on them."""
    g = _gen(seed)
    X = torch.randn(n, 13, generator=g, device=DEV) * torch.logspace(-1, 1, 13, device=DEV) + 0.3
    M = torch.randn(13, 9, generator=g, device=DEV) / 13
    T = 0.01 * torch.tanh(X / X.std(0) @ M) + 0.002 * torch.randn(n, 9, generator=g, device=DEV)
    return X, T


def _weights(seed):
    """Closure parameters of the size training leaves, and their normalisation."""
    g = _gen(seed + 99)
    lim = [math.sqrt(6 / 77)] * 832 + [0.1] * 64 + [math.sqrt(6 / 128)] * 4096 + [0.1] * 64 + [math.sqrt(6 / 73)] * 576 + [0.1] * 9
    w = (torch.rand(len(lim), generator=g, device=DEV) * 2 - 1) * torch.tensor(lim, device=DEV)
    sd = torch.tensor([1.0, 1.0, 2.0] * 3 + [1.0, 1.0, 2.0] + [60.0], device=DEV)
    norm = torch.cat([torch.zeros(12, device=DEV), torch.full((1,), 80.0, device=DEV), sd, torch.zeros(9, device=DEV),
                      torch.full((9,), 2e-4, device=DEV)])
    return w.cpu().numpy(), norm.cpu().numpy()


def _pinned(shape):
    return torch.empty(shape, dtype=F64, pin_memory=True).numpy()


def _slip(p):
    return spanwise_stripes(p.nP, 6, Tw=p.Tw[0])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        chans, outs = [], []
        for p, mesh, var, Ri in _members(case, seed):
            ch = Channel(p, *mesh)
            ch.set_buoyancy(Ri, 1.0)
            ch.init_sol_v(var.cpu().numpy())
            chans.append(ch)
            outs.append(_pinned(ch.shape))
        return dict(case=case, ens=Ensemble(chans), chans=chans, outs=outs)
    if kind == "train":
        X, T = _features(case["n"], seed)
        cl = Closure(capacity=case["n"])
        cl.add_data(X.cpu().numpy(), T.cpu().numpy())
        cl.fit_normalization()
        cl.init(seed=seed)
        return dict(case=case, cl=cl, seed=seed)
    if kind == "infer":
        cl = Closure()
        w, norm = _weights(seed)
        cl.norm, cl.params = norm, w
        X = torch.randn(case["n"], 13, generator=_gen(seed), device=DEV).cpu().numpy()
        return dict(case=case, cl=cl, X=X * norm[13:26] + norm[:13])
    p, mesh, var = _flow(case, seed)
    host = var.cpu().numpy()
    ch = Channel(p, *mesh)
    s = dict(case=case, ch=ch, var=host)
    if kind != "restart":
        ch.init_sol_v(host)
    if kind in ("steps", "closure_run"):
        s["out"] = _pinned(ch.shape)
    if case.get("wall") == "slip":
        ch.set_wall_bc(0, _slip(p))
        ch.set_wall_bc(1, WallBC(Tw=p.Tw[1]))
    if case.get("diag"):
        ch.diag_enable(planes=PLANES, every=case["diag"])
    if kind == "closure_run":
        cl = Closure()
        w, norm = _weights(seed)
        cl.norm, cl.params = norm, w
        s["cl"] = cl
        attach(ch, cl, True, every_stage=not case["hold"])
    if kind == "sample":
        ch.calc_tau_wall()
        ch.avg_spatial()
        n = ((p.nP[0] - 3) // case["sx"] + 1) * ((p.nP[1] - 3) // case["sy"] + 1) * ((p.nP[2] - 1) // case["sz"] - 1)
        s["n"] = n
    if kind == "post":
        ch.avg_spatial()
        s["mean"] = ch.stats()[1]
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind in ("steps", "closure_run", "restart"):
        ch = s["ch"]
        if kind == "restart":
            ch.init_sol_v(s["var"])
        ch.step(case["steps"])
        tau, s1, s2, c = ch.stats()
        r = dict(tau=tau, s1=s1, s2=s2, corr=c, var=ch.download(s.get("out")))
        if case.get("diag"):
            d = ch.diag_read()
            r["diag"] = {k: d[k] for k in ("time", "ke", "rho_b", "u_b", "rhou_b")}
        return r
    if kind == "sweep":
        s["ens"].step(case["steps"])
        return [dict(s1=ch.stats()[1], var=ch.download(o)) for ch, o in zip(s["chans"], s["outs"])]
    if kind == "train":
        losses = s["cl"].train(1, batch=case["batch"], lr=1e-3, seed=s["seed"])
        return dict(losses=losses, params=s["cl"].params)
    if kind == "infer":
        return s["cl"].infer(s["X"])
    if kind == "sample":
        with Closure(capacity=s["n"]) as cl:
            cl.sample(s["ch"], strides=(case["sx"], case["sy"], case["sz"]), width=case["width"])
            norm = cl.fit_normalization()
            X, T = cl.data()
        return dict(X=X, T=T, norm=norm)
    fluc, q = s["ch"].fluctuation_q(s["mean"])
    return dict(fluc=fluc, q=q)


# --------------------------------------------------------------------- work
FLOPS_STAGE = 420        # arithmetic of one point's stage: conversion, fluxes in three directions, update
FLOPS_MLP = 2 * (13 * 64 + 64 * 64 + 64 * 9)


def work(case):
    """Each stage reads its input and (after the first) the step's base state, and writes its output."""
    kind = case["kind"]
    if kind == "sweep":
        n = sum((q[0] - 2) * (q[1] - 2) * (q[2] - 2) for q in _sweep_grids(case))
        by = (240 if case["mixed"] else 320) * n * case["steps"] + 112 * n
        return {"bytes": by, "flops": 3 * FLOPS_STAGE * n * case["steps"]}
    if kind == "train":
        rows = case["n"] // case["batch"] * case["batch"]
        return {"bytes": 88 * rows, "flops": 3 * FLOPS_MLP * rows}
    if kind == "infer":
        return {"bytes": 88 * case["n"], "flops": FLOPS_MLP * case["n"]}
    n = (case["n1"] - 2) * (case["n2"] - 2) * (case["n3"] - 2)
    if kind == "sample":
        m = n // (case["sx"] * case["sy"] * case["sz"])
        taps = (case["width"] + 1) ** 2
        return {"bytes": 40 * n + 88 * m, "flops": 60.0 * taps * n}
    if kind == "post":
        return {"bytes": 40 * n + 64 * n, "flops": 90 * n}
    rk = case.get("rk", 3)
    per = {(2, False): 200, (3, False): 320, (2, True): 160, (3, True): 240}[rk, case.get("mixed", False)]
    steps = case["steps"]
    by, fl = per * n * steps + 112 * n, rk * FLOPS_STAGE * n * steps
    if kind == "closure_run":
        evals = steps * (1 if case["hold"] else 3)
        by, fl = by + evals * n * (40 + 4 * 40), fl + evals * n * (FLOPS_MLP + 120)
    if kind == "restart":
        by += 40 * n
    return {"bytes": by, "flops": fl}


def _sweep_grids(case):
    n, lo, hi = case["members"], case["lo"], case["hi"]
    for c in range(n):
        f = [((c * s) % n) / max(n - 1, 1) for s in (1, 5, 3)]
        yield lo + round(f[0] * (hi - lo)), lo + round(f[1] * 0.67 * (hi - lo)), lo + 1 + round(f[2] * 0.67 * (hi - lo))


# ------------------------------------------------ the same in 64 bits (torch)
class _Exact:
    """The solver's equations on the unique periodic points, with the walls' stored points."""

    def __init__(self, p, mesh, var, slip=None, Ri=0.0, closure=None, hold=True):
        self.p, (self.x3, self.jac, self.inv) = p, mesh
        self.slip, self.Ri, self.closure, self.hold = slip, Ri, closure, hold
        n1, n2, n3 = p.nP
        self.n1, self.n2, self.n3 = n1, n2, n3
        k3 = lambda a: torch.tensor(np.array(a), device=DEV, dtype=F64)[:, None, None]  # noqa: E731
        self.zinv, self.zjac = k3(self.inv / p.dXi), k3(self.jac)
        c = slice(1, -1)
        prim = var[:, :, c, c]
        self.Q = torch.cat([prim[:1], prim[:1] * prim[1:5]])
        self.wall = [var[:, k].clone() for k in (0, n3 - 1)]         # full stored points, 7 variables
        self.edge = var[:, :, ::n2 - 1, ::n1 - 1].clone()            # the stale corner columns
        self.tau, self.rhobar = [0.0, 0.0], torch.zeros(n3, 1, 1, device=DEV, dtype=F64)
        self.steps_done, self.diag = 0, []
        self.stats = [torch.zeros(r, n3, device=DEV, dtype=F64) for r in (7, 7, 9)]
        x = self.x3
        self.one = []                                                # one-sided first / second derivatives
        for a, b, d in ((x[0], x[1], x[2]), (x[-1], x[-2], x[-3])):
            h1, h2 = b - a, d - a
            self.one.append((-(h1 + h2) / (h1 * h2), h2 / (h1 * (h2 - h1)), -h1 / (h2 * (h2 - h1)),
                             -2 / (h1 * (h2 - h1)), 2 / (h2 * (h2 - h1))))
        self._prims()

    def _prims(self):
        p, c = self.p, slice(1, -1)
        r = self.Q[0].clone()
        u, v, w, E = (self.Q[m] / r for m in (1, 2, 3, 4))
        T = E - 0.5 * p.ggM * (u * u + v * v + w * w)
        P = r * T / (p.gama * p.Mac ** 2)
        for k, W in ((0, self.wall[0]), (-1, self.wall[1])):
            for a, m in ((r, 0), (u, 1), (v, 2), (w, 3), (E, 4), (T, 5), (P, 6)):
                a[k] = W[m][c, c]
        self.prim = [r, u, v, w, E, T, P]

    def _hybrid(self, vel, sh, cond, inv):
        e, w = 0.5 * (vel + sh(vel, 1)), 0.5 * (vel + sh(vel, -1))
        v1, vm1, v2, vm2 = (sh(vel, o) for o in (1, -1, 2, -2))
        out = []
        for m in range(5):
            q0 = self.Q[m]
            q1, qm, q2, qm2 = (sh(q0, o) for o in (1, -1, 2, -2))
            quick = e * torch.where(e >= 0, 6 * q0 + 3 * q1 - qm, 6 * q1 + 3 * q0 - q2) \
                - w * torch.where(w >= 0, 6 * qm + 3 * q0 - qm2, 6 * q0 + 3 * qm - q1)
            cent = 8 * (v1 * q1 - vm1 * qm) - v2 * q2 + vm2 * qm2
            out.append(torch.where(cond, quick * (inv / 8), cent * (inv / 12)))
        return out

    def stage(self, base, a, b, cdt, S):
        p, n3 = self.p, self.n3
        r, u, v, w, E, T, P = self.prim
        mu = T.pow(0.7)
        rx = lambda f, o: torch.roll(f, -o, -1)  # noqa: E731
        ry = lambda f, o: torch.roll(f, -o, -2)  # noqa: E731
        rz = lambda f, o: torch.roll(f, -o, 0)   # noqa: E731  (the ends are overwritten below)
        idx, idy = 1 / p.dx, 1 / p.dy
        flux = self._hybrid(u, rx, p.Re * self.Q[1].abs() * p.dx / mu > p.Pe[0], idx)
        for m, f in enumerate(self._hybrid(v, ry, p.Re * self.Q[2].abs() * p.dy / mu > p.Pe[1], idy)):
            flux[m] += f
        for m, f in enumerate(self._hybrid(w, rz, p.Re * self.Q[3].abs() * p.dXi * self.zjac / mu > p.Pe[2], self.zinv)):
            g = w * self.Q[m]
            for k in (1, n3 - 2):
                f[k] = (g[k + 1] - g[k - 1]) * (0.5 * self.zinv[k])
            flux[m] += f
        dx = lambda f: (rx(f, 1) - rx(f, -1)) * (0.5 * idx)  # noqa: E731
        dy = lambda f: (ry(f, 1) - ry(f, -1)) * (0.5 * idy)  # noqa: E731

        def dz(f):
            d = (rz(f, 1) - rz(f, -1)) * (0.5 * self.zinv)
            d[0] = (f[1] - f[0]) / (self.x3[1] - self.x3[0])
            d[-1] = (f[-1] - f[-2]) / (self.x3[-1] - self.x3[-2])
            return d

        G = [[d(f) for d in (dx, dy, dz)] for f in (u, v, w, T)]
        c = slice(1, -1)
        for k, W in ((0, self.wall[0]), (-1, self.wall[1])):         # a wall's own neighbours, duplicates included
            for m in range(3):
                G[m][0][k] = (W[m + 1][c, 2:] - W[m + 1][c, :-2]) * (0.5 * idx)
                G[m][1][k] = (W[m + 1][2:, c] - W[m + 1][:-2, c]) * (0.5 * idy)
        mr, div = mu / p.Re, G[0][0] + G[1][1] + G[2][2]
        vel = (u, v, w)
        for d, dd in ((0, dx), (1, dy), (2, dz)):
            col = [-(mr * (G[m][d] + G[d][m])) + (P + 2 / 3 * mr * div if m == d else 0) for m in range(3)]
            heat = -p.gama / p.Pr * mr * G[3][d] + p.ggM * sum(vel[m] * col[m] for m in range(3))
            for m, f in enumerate(col + [heat]):
                flux[m + 1] += dd(f)
        force = 0.5 * (self.tau[0] - self.tau[1]) * self.rhobar
        src = [0.0, force, 0.0, 0.0, p.ggM * u * force]
        if self.Ri:
            bq = self.Ri * r * (T - 1.0)
            src[3], src[4] = bq, src[4] + p.ggM * w * bq
        new = self.Q.clone()
        for m in range(5):
            R = src[m] - flux[m]
            if S is not None and m:
                R = R + S[m - 1]
            new[m, 1:-1] = (a * base[m] + b * self.Q[m] + cdt * R)[1:-1]
        self.Q = new
        self._prims()
        self._walls()

    def _walls(self):
        p, c = self.p, slice(1, -1)
        for side, W in enumerate(self.wall):
            k2, k3 = (1, 2) if side == 0 else (-2, -3)
            c0, c1, c2, e1, e2 = self.one[side]
            f2, f3 = ([_full(a[k]) for a in self.prim] for k in (k2, k3))
            for f, k in ((f2, k2), (f3, k3)):
                for m in range(7):
                    f[m][::self.n2 - 1, ::self.n1 - 1] = self.edge[m, k]
            W[1:4] = 0
            W[5] = p.Tw[side]
            if self.slip is not None and side == 0:
                for m in (1, 2):
                    W[m] = torch.where(self.slip, -(c1 * f2[m] + c2 * f3[m]) / c0, 0.0)
            W[4] = W[5] + 0.5 * p.ggM * (W[1] ** 2 + W[2] ** 2)
            W[0] = p.gama * p.Mac ** 2 * W[6] / W[5]
            mu, mu2, mu3 = W[5].pow(0.7), f2[5].pow(0.7), f3[5].pow(0.7)
            gu, gv = (c0 * mu * W[m] + c1 * mu2 * f2[m] + c2 * mu3 * f3[m] for m in (1, 2))
            dux = (gu[c, 2:] - gu[c, :-2]) * (0.5 / p.dx)
            dvy = (gv[2:, c] - gv[:-2, c]) * (0.5 / p.dy)
            d2w = (e1 * mu2 * f2[3] + e2 * mu3 * f3[3])[c, c]
            rw2 = (c1 * f2[0] * f2[3] ** 2 + c2 * f3[0] * f3[3] ** 2)[c, c]
            lhs = (-dux - dvy + 2 / 3 * (dux + dvy - 2 * d2w)) / p.Re + rw2
            W[6][c, c] = -(lhs + (c1 * f2[6] + c2 * f3[6])[c, c]) / c0
        self._prims()

    def var(self):
        out = _full(torch.stack(self.prim))
        out[:, 1:-1, ::self.n2 - 1, ::self.n1 - 1] = self.edge[:, 1:-1]
        out[:, 0], out[:, -1] = self.wall
        return out

    def moments(self, tau=True, planes=True):
        p, V, c = self.p, self.var(), slice(1, -1)
        if tau:
            for side, k in enumerate(((0, 1, 2), (-1, -2, -3))):
                mu = V[5, k[0]].pow(0.7)[c, c]
                du = sum(self.one[side][m] * V[1, k[m]][c, c] for m in range(3))
                dw = (V[3, k[0]][c, 2:] - V[3, k[0]][c, :-2]) * (0.5 / p.dx)
                self.tau[side] = float((mu * (du + dw)).mean() / p.Re)
        if planes:
            pairs = ((0, 3), (0, 5), (1, 2), (1, 3), (2, 3), (2, 5), (5, 3), (6, 3), (6, 5))
            self.stats = [V.mean((2, 3)), (V * V).mean((2, 3)), torch.stack([(V[a] * V[b]).mean((1, 2)) for a, b in pairs])]
            self.rhobar = self.stats[0][0][:, None, None]
        return V

    def series(self, time):
        p, V = self.p, self.var()
        area = torch.tensor(np.diff(self.x3), device=DEV, dtype=F64)[:, None] * p.dy
        cell = lambda f: ((f[:-1, :-1] + f[:-1, 1:] + f[1:, :-1] + f[1:, 1:]) * 0.25 * area).sum() / (self.x3[-1] * p.Ly)  # noqa: E731
        rec = [[], [], []]
        for i in PLANES:
            ok = 2 < i < self.n1 - 1
            r, u = V[0, :, :, i - 1], V[1, :, :, i - 1]
            for q, f in enumerate((r, u, r * u)):
                rec[q].append(float(cell(f)) if ok else 0.0)
        self.diag.append((time, float((V[1:4] ** 2).sum(0).mean()), *rec))

    def advance(self, steps, diag=0):
        p, time = self.p, 0.0
        coef = [(0, 1, 1), (.75, .25, .25), (1 / 3, 2 / 3, 2 / 3)] if p.rk_scheme == 3 else [(0, 1, .5), (1, 0, 1)]
        for n in range(1, steps + 1):
            base, S = self.Q, None
            for i, (a, b, cc) in enumerate(coef):
                if self.closure is not None and (i == 0 or not self.hold):
                    S = self._closure_source()
                self.stage(base, a, b, cc * p.dt, S)
            time += p.dt
            if diag and n % diag == 0:
                self.series(time)
            if n % p.istat == 0:
                self.moments()
        return self

    # learned closure: features, network, divergence
    def filtered(self, width):
        r, u, v, w, _, T, _ = self.prim
        f = [r, r * u, r * v, r * w, r * T, r * u * u, r * v * v, r * w * w, r * u * v, r * u * w, r * v * w,
             r * u * T, r * v * T, r * w * T]
        h = width // 2
        if h:
            wt = {o: (0.5 if abs(o) == h else 1.0) / width for o in range(-h, h + 1)}
            for d in (-1, -2):
                f = [sum(wt[o] * torch.roll(a, -o, d) for o in wt) for a in f]
        return f

    def features(self, sx, sy, sz, width, targets):
        p, n3 = self.p, self.n3
        f = self.filtered(width)
        r, (u, v, w, T) = f[0], (a / f[0] for a in f[1:5])
        kk = torch.arange(n3, device=DEV)
        kp, km = (kk + sz).clamp(max=n3 - 1), (kk - sz).clamp(min=0)
        z = torch.tensor(self.x3, device=DEV, dtype=F64)
        X = []
        for a in (u, v, w, T):
            X.append((torch.roll(a, -sx, -1) - torch.roll(a, sx, -1)) / (2 * sx * p.dx))
            X.append((torch.roll(a, -sy, -2) - torch.roll(a, sy, -2)) / (2 * sy * p.dy))
            X.append((a[kp] - a[km]) / (z[kp] - z[km])[:, None, None])
        rw = 0.5 * float(self.stats[0][0, 0] + self.stats[0][0, -1])
        ut = math.sqrt(max(0.5 * (self.tau[0] - self.tau[1]), 0.0) / rw) if rw > 0 else 0.0
        muw = 0.5 * (p.Tw[0] ** 0.7 + p.Tw[1] ** 0.7)
        yp = rw * ut * torch.minimum(z - z[0], z[-1] - z) * p.Re / muw
        X = torch.stack(X + [yp[:, None, None] + 0 * r])
        X = X[:, sz:sz + ((n3 - 1) // sz - 1) * sz:sz, ::sy, ::sx].permute(1, 2, 3, 0).reshape(-1, 13)
        if not targets:
            return X
        Y = [f[5] - r * u * u, f[6] - r * v * v, f[7] - r * w * w, f[8] - r * u * v, f[9] - r * u * w, f[10] - r * v * w,
             f[11] - r * u * T, f[12] - r * v * T, f[13] - r * w * T]
        Y = torch.stack(Y)[:, sz:sz + ((n3 - 1) // sz - 1) * sz:sz, ::sy, ::sx].permute(1, 2, 3, 0).reshape(-1, 9)
        return X, Y

    def _closure_source(self):
        p = self.p
        Y = _mlp(*self.closure, self.features(1, 1, 1, 0, False))[0]
        m1, m2, m3 = self.n1 - 2, self.n2 - 2, self.n3
        F = torch.zeros(9, m3, m2, m1, device=DEV, dtype=F64)
        F[:, 1:-1] = Y.T.reshape(9, m3 - 2, m2, m1)
        S = []
        for a, (cx, cy, cz) in enumerate(((0, 3, 4), (3, 1, 5), (4, 5, 2), (6, 7, 8))):
            d = (torch.roll(F[cx], -1, -1) - torch.roll(F[cx], 1, -1)) * (0.5 / p.dx) \
                + (torch.roll(F[cy], -1, -2) - torch.roll(F[cy], 1, -2)) * (0.5 / p.dy) \
                + (torch.roll(F[cz], -1, 0) - torch.roll(F[cz], 1, 0)) * (0.5 * self.zinv)
            S.append(-d if a < 3 else -p.gama * d)
        return S


def _unpack(w):
    o, out = 0, []
    for shape in ((64, 13), (64,), (64, 64), (64,), (9, 64), (9,)):
        n = math.prod(shape)
        out.append(w[o:o + n].view(shape))
        o += n
    return out


def _mlp(w, norm, X):
    """Outputs in physical and in normalised units."""
    W1, b1, W2, b2, W3, b3 = _unpack(w)
    gelu = lambda z: torch.nn.functional.gelu(z, approximate="tanh")  # noqa: E731
    h = gelu(((X - norm[:13]) / norm[13:26]) @ W1.T + b1)
    y = gelu(h @ W2.T + b2) @ W3.T + b3
    return y * norm[35:] + norm[26:35], y


def _hash(x):
    m = (1 << 64) - 1
    x = (x + 0x9E3779B97F4A7C15) & m
    z = x
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return x, z ^ (z >> 31)


def _norm_of(X, T):
    sd = lambda a: a.std(0, unbiased=False)  # noqa: E731
    return torch.cat([X.mean(0), sd(X), T.mean(0), sd(T)])


def _exact_train(case, seed):
    X, T = (a.to(F64) for a in _features(case["n"], seed))
    norm = _norm_of(X, T)
    st, w = seed, []
    for n, fan in ((832, 77), (64, 0), (4096, 128), (64, 0), (576, 73), (9, 0)):
        for _ in range(n):
            h = 0
            if fan:
                st, h = _hash(st)
            w.append(((h >> 11) / 2 ** 53 * 2 - 1) * math.sqrt(6 / fan) if fan else 0.0)
    w = torch.tensor(w, device=DEV, dtype=torch.float32).to(F64).requires_grad_()
    n, batch = case["n"], case["batch"]
    st, a = _hash(seed)
    a = a % n | 1
    while math.gcd(a, n) != 1:
        a = (a + 2) % n
    st, b = _hash(st)
    b %= n
    m, v, loss = torch.zeros_like(w), torch.zeros_like(w), 0.0
    for t in range(1, n // batch + 1):
        rows = (a * torch.arange((t - 1) * batch, t * batch, device=DEV) + b) % n
        e = _mlp(w, norm, X[rows])[1] - (T[rows] - norm[26:35]) / norm[35:]
        l = (e * e).mean()
        g, = torch.autograd.grad(l, w)
        loss += float(l.detach()) / (n // batch)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        w = (w - 1e-3 * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)).detach().requires_grad_()
    return dict(losses=torch.tensor([loss], dtype=F64), params=w.detach())


def exact(case, seed):
    kind = case["kind"]
    if kind == "sweep":
        out = []
        for p, mesh, var, Ri in _members(case, seed):
            e = _Exact(p, mesh, var, Ri=Ri).advance(case["steps"])
            out.append(dict(s1=e.stats[0], var=e.var()))
        return out
    if kind == "train":
        return _exact_train(case, seed)
    weights = [torch.tensor(a, device=DEV, dtype=F64) for a in _weights(seed)]
    if kind == "infer":
        X = torch.randn(case["n"], 13, generator=_gen(seed), device=DEV)
        X = X * weights[1][13:26].float() + weights[1][:13].float()
        return _mlp(*weights, X.to(F64))[0]
    p, mesh, var = _flow(case, seed)
    slip = torch.tensor(_slip(p).mask != 0, device=DEV) if case.get("wall") == "slip" else None
    e = _Exact(p, mesh, var, slip=slip, closure=weights if kind == "closure_run" else None, hold=case.get("hold", True))
    if kind in ("sample", "post"):
        V = e.moments()
        if kind == "sample":
            X, T = e.features(case["sx"], case["sy"], case["sz"], case["width"], True)
            return dict(X=X, T=T, norm=_norm_of(X, T))
        fluc = V - e.stats[0][:, :, None, None]
        return dict(fluc=fluc, q=_q_criterion(fluc[1:4], p, mesh[0]))
    e.advance(case["steps"], case.get("diag", 0))
    r = dict(tau=torch.tensor(e.tau, dtype=F64), s1=e.stats[0], s2=e.stats[1], corr=e.stats[2], var=e.var())
    if case.get("diag"):
        rec = list(zip(*e.diag)) or [[]] * 5
        keys = ("time", "ke", "rho_b", "u_b", "rhou_b")
        r["diag"] = {k: torch.tensor(rec[i], dtype=F64).reshape((-1,) if i < 2 else (-1, len(PLANES)))
                     for i, k in enumerate(keys)}
    return r


def _q_criterion(vel, p, x3):
    grid = [torch.arange(p.nP[0], device=DEV, dtype=F64) * p.dx, torch.arange(p.nP[1], device=DEV, dtype=F64) * p.dy,
            torch.tensor(x3, device=DEV, dtype=F64)]
    J = [[None] * 3 for _ in range(3)]
    for c in range(3):
        for b, dim in enumerate((2, 1, 0)):
            d = grid[b].diff().view([-1 if k == dim else 1 for k in range(3)])
            n = vel[c].shape[dim]
            s = vel[c].diff(dim=dim)
            d1, d2 = d.narrow(dim, 1, n - 2), d.narrow(dim, 0, n - 2)
            g = (d2 / d1 * s.narrow(dim, 1, n - 2) + d1 / d2 * s.narrow(dim, 0, n - 2)) / (d1 + d2)
            for o in range(3):
                if o != dim:
                    g = g.narrow(o, 1, g.shape[o] - 2)
            J[c][b] = g
    tr = J[0][0] + J[1][1] + J[2][2]
    ss = sum(J[a][b] * J[b][a] for a in range(3) for b in range(3))   # sum S^2 - sum R^2 (R antisymmetric)
    q = torch.zeros(vel.shape[1:], device=DEV, dtype=F64)
    q[1:-1, 1:-1, 1:-1] = 0.5 * (tr * tr - ss)
    return q
