"""Performance cases: the work that a user of the framework has it do, through its public
entry points, over the range of sizes, stencil orders, precisions and time schemes in use.

A case is a dict of plain values; `listed()` names the standing ones and `draw(rng)` gives
more of the same ranges. `prepare(case, seed)` makes what a program holds before the call
(page-locked host fields, the solver / batch / server handle), `run(state)` is one pass.

Kinds of pass
  run    one leg of a simulation between two outputs, as the reference's main loop does it:
         set the fields (copyField(0)), set the clock, advance `steps` time steps, fetch the
         fields and the per-step logs (copyField(1))
  rhs    one evaluation of the right-hand side of the fields held by the solver
  batch  `steps` steps of an ensemble and its members' fields; the members go on from pass
         to pass, as a parameter sweep does
  serve  a wave of "advance N steps" requests submitted to a server and awaited
  stats  the flow statistics printed at every output: dissipation and enstrophy, plane
         profiles, friction Reynolds number
"""
from __future__ import annotations

import math

import numpy as np
import torch

from cudanavierstokes_gb300 import (PREC_FP32_RHS, PREC_FP64, PREC_PAIR_RHS, RK3_CLASSIC, RK3_LOWSTORAGE, RK4_CLASSIC,
                                    Solver, boundary_layer_params, channel_params, tgv_params)
from cudanavierstokes_gb300.batch import Batch
from cudanavierstokes_gb300.roofline import STAGE_BYTES, stage_flops
from cudanavierstokes_gb300.server import Server

PREC = {"fp64": PREC_FP64, "fp32": PREC_FP32_RHS, "pair": PREC_PAIR_RHS}
SCHEME = {"ls": RK3_LOWSTORAGE, "rk3": RK3_CLASSIC, "rk4": RK4_CLASSIC}


# ---------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------
def _run(flow, mx, my, mz, prec, steps, S=4, V=4, scheme="ls", Re=0.0, Ma=0.0):
    return dict(kind="run", flow=flow, mx=mx, my=my, mz=mz, S=S, V=V, prec=prec, scheme=scheme, steps=steps, Re=Re,
                Ma=Ma)


def listed():
    return [
        # a first try of a set-up on a toy box: launches and latency count, not arithmetic
        dict(name="tgv_fp64_16x20x24", **_run("tgv", 16, 20, 24, "fp64", 10)),
        # the standard Taylor-Green validation box
        dict(name="tgv_fp64_64", **_run("tgv", 64, 64, 64, "fp64", 20)),
        # the benchmark channel (supersonic, isothermal walls, body force), plain FP64
        dict(name="channel_fp64_128x160x192", **_run("channel", 128, 160, 192, "fp64", 10)),
        # the same channel with the RHS in pairs and in FP32
        dict(name="channel_pair_128x160x192", **_run("channel", 128, 160, 192, "pair", 10)),
        dict(name="channel_fp32_128x160x192", **_run("channel", 128, 160, 192, "fp32", 20)),
        # the largest: a production decay run
        dict(name="tgv_fp32_256", **_run("tgv", 256, 256, 256, "fp32", 10)),
        # a spatial boundary layer: sponge, wall perturbation, extrapolated ends, lower orders
        dict(name="bl_fp64_s3v2_72x20x320", **_run("bl", 72, 20, 320, "fp64", 10, S=3, V=2)),
        # odd edges, mixed orders, the classic RK3
        dict(name="tgv_fp64_s4v2_rk3_75x53x91", **_run("tgv", 75, 53, 91, "fp64", 10, V=2, scheme="rk3")),
        # one RHS evaluation, as a coupling or an implicit outer loop asks for
        dict(name="rhs_channel_fp64_64x48x64", kind="rhs", flow="channel", mx=64, my=48, mz=64, S=4, V=4, prec="fp64"),
        # a Taylor-Green ensemble (Reynolds and Mach sweep), all members together
        dict(name="batch_fp32_8", kind="batch", members=8, prec="fp32", steps=20, lo=32, hi=128),
        # a wave of requests of mixed sizes on a server
        dict(name="serve_fp32_6", kind="serve", requests=6, prec="fp32", steps=80, lo=32, hi=96),
        # the statistics of an output of the benchmark channel
        dict(name="stats_channel_128x160x192", kind="stats", flow="channel", mx=128, my=160, mz=192, S=4, V=4,
             prec="fp64"),
    ]


def _edge(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _orders(rng):
    S = rng.choice((4, 4, 4, 4, 3, 3, 2, 1))
    return S, (S if rng.random() < 0.6 else rng.randint(1, S))


def draw(rng):
    what = rng.choices(("run", "rhs", "batch", "serve", "stats"), (60, 12, 9, 9, 10))[0]
    if what == "batch":
        return dict(kind="batch", members=rng.randint(2, 12), prec=rng.choice(("fp32", "fp32", "fp64")),
                    steps=rng.randint(5, 20), lo=24, hi=rng.choice((48, 64, 96)))
    if what == "serve":
        return dict(kind="serve", requests=rng.randint(2, 6), prec="fp32", steps=rng.randint(20, 80), lo=24,
                    hi=rng.choice((48, 64, 96)))
    flow = rng.choices(("tgv", "channel", "bl"), (45, 40, 15))[0]
    S, V = _orders(rng)
    prec = rng.choices(("fp64", "fp32", "pair"), (50, 35, 15))[0]
    if flow == "bl":
        mx, my, mz = _edge(rng, 24, 96), _edge(rng, 12, 48), _edge(rng, 144, 480)
    else:
        mx, my, mz = _edge(rng, 14, 200), _edge(rng, 14, 200), _edge(rng, 14, 200)
    c = dict(flow=flow, mx=mx, my=my, mz=mz, S=S, V=V, prec=prec)
    if what in ("rhs", "stats"):
        return dict(kind=what, **c)
    scheme = rng.choices(("ls", "rk3", "rk4"), (70, 15, 15))[0]
    steps = max(1, min(rng.randint(2, 30), int((4e7 if prec == "fp64" else 1.2e8) / (mx * my * mz))))
    Re = round(math.exp(rng.uniform(math.log(400.0), math.log(3200.0))), 3) if flow != "bl" else 0.0
    Ma = round(rng.uniform(0.1, 0.8), 4) if flow == "tgv" else 0.0
    return dict(kind="run", scheme=scheme, steps=steps, Re=Re, Ma=Ma, **c)


def _params(c):
    make = {"tgv": tgv_params, "channel": channel_params, "bl": boundary_layer_params}[c["flow"]]
    p = make().copy(mx=c["mx"], my=c["my"], mz=c["mz"], stencil_size=c["S"], stencil_visc=c["V"],
                    precision=PREC[c["prec"]])
    if c.get("scheme"):
        p = p.copy(scheme=SCHEME[c["scheme"]])
    if c.get("Re"):
        p = p.copy(Re=c["Re"])
    if c.get("Ma"):
        p = p.copy(Ma=c["Ma"])
    return p


def _ensemble(c, seed):
    """The members of a batch or the requests of a wave: Taylor-Green boxes (edge, Re and Ma
    drawn) and, served, every third a small stretched channel. Sizes are the case's, the
    physics the seed's."""
    sizes = np.random.default_rng(1000 + c[("members" if c["kind"] == "batch" else "requests")])
    rng = np.random.default_rng(seed)
    out = []
    for q in range(c["members"] if c["kind"] == "batch" else c["requests"]):
        edges = [e for e in (24, 32, 48, 64, 96, 128) if c["lo"] <= e <= c["hi"]]
        edge = int(sizes.choice(edges))
        if c["kind"] == "serve" and q % 3 == 2:
            p = channel_params(64, 48, 64, precision=PREC[c["prec"]])
        else:
            p = tgv_params(edge, precision=PREC[c["prec"]], Re=float(math.exp(rng.uniform(math.log(400), math.log(1600)))),
                           Ma=float(rng.uniform(0.1, 0.8)))
        out.append((p, int(rng.integers(1 << 30))))
    return out


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _grid(p):
    """Cell-centred coordinates and metrics of the framework's grid: x (tanh-stretched where
    asked for), xp = 1/x'(xi), xpp = x''(xi), y, z, as numpy."""
    mx, S = p.mx, p.stencil_size
    cF, cS = _weights(S)
    dx = p.Lx / mx
    denom, denom2 = (2 * mx, 1.0) if p.boundary_layer else (mx, 2.0)
    xn = np.tanh(p.stretch * (np.arange(mx + 1) / denom - 0.5)) / math.tanh(p.stretch * 0.5)
    x = p.Lx * (1.0 + (xn[:-1] + xn[1:]) / 2.0) / denom2
    fb = np.concatenate([-x[:S][::-1], x, 2 * p.Lx - x[-S:][::-1]])
    xp = sum(cF[k] * (fb[S + k:S + k + mx] - fb[S - k:S - k + mx]) for k in range(1, S + 1)) / dx
    xpp = (cS[0] * x + sum(cS[k] * (fb[S + k:S + k + mx] + fb[S - k:S - k + mx]) for k in range(1, S + 1))) / dx / dx
    if not p.nonuniform_x:
        x = p.Lx * (0.5 + np.arange(mx)) / mx
    y = p.Ly * (0.5 + np.arange(p.my)) / p.my
    z = p.Lz * (0.5 + np.arange(p.mz)) / p.mz
    return x, 1.0 / xp, xpp, y, z


def _weights(n):
    """Central first- and second-derivative weights of order 2n: c1[1..n], c2[0..n]."""
    return {1: ([0, 1 / 2], [-2.0, 1.0]),
            2: ([0, 2 / 3, -1 / 12], [-5 / 2, 4 / 3, -1 / 12]),
            3: ([0, 3 / 4, -3 / 20, 1 / 60], [-49 / 18, 3 / 2, -3 / 20, 1 / 90]),
            4: ([0, 4 / 5, -1 / 5, 4 / 105, -1 / 280], [-205 / 72, 8 / 5, -1 / 5, 8 / 315, -1 / 560])}[n]


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _noise(shape, seed, amp):
    g = torch.Generator(device="cpu").manual_seed(seed)
    return ((torch.rand(shape, generator=g, dtype=torch.float64) * 2 - 1) * amp).to(_dev())


def _bl_refs(p):
    """Boundary-layer reference fields on the (z, x) plane: a growing tanh profile with a warm
    wall, and the sponge strengths on x and z."""
    x, _, _, _, z = _grid(p)
    Rgas = 1.0 / (p.gam * p.Ma * p.Ma)
    d = np.sqrt(1.0 + z / p.Re)[:, None]
    w = np.tanh(1.3 * x[None, :] / d)
    T = 1.0 + 0.02 * (1.0 - w * w)
    r = 1.0 / T
    u = 0.4 * w * w / (d * p.Re)
    e = r * Rgas * T / (p.gam - 1.0) + 0.5 * r * (u * u + w * w)
    sx = np.where(x >= p.Lx - p.sp_top_len, p.sp_top_str * np.abs((x - (p.Lx - p.sp_top_len)) / p.sp_top_len) ** p.sp_top_exp, 0.0)
    sz = np.where(z <= p.sp_inl_len, p.sp_inl_str * np.abs((p.sp_inl_len - z) / p.sp_inl_len) ** p.sp_inl_exp, 0.0)
    sz = np.where(z >= p.Lz - p.sp_out_len, p.sp_out_str * np.abs((z - (p.Lz - p.sp_out_len)) / p.sp_out_len) ** p.sp_out_exp, sz)
    return [np.ascontiguousarray(a) for a in (sx, sz, r, u, w, e)]


def _fields(p, seed, flow, developed=False):
    """Initial rho, u, v, w, rhoE of shape (mz, my, mx) as float64 tensors; `developed` adds
    density waves and velocity noise, as a flow has them some time after such a start."""
    x, _, _, y, z = (torch.tensor(a, device=_dev()) for a in _grid(p))
    Rgas = 1.0 / (p.gam * p.Ma * p.Ma)
    shape = (p.mz, p.my, p.mx)
    one = torch.ones(shape, dtype=torch.float64, device=_dev())
    if flow == "tgv":      # Taylor-Green vortex with per-axis phase offsets
        ph = np.random.default_rng(seed).uniform(0.0, 2 * math.pi, size=3)
        X = (2 * math.pi * x / p.Lx + ph[0])[None, None, :]
        Y = (2 * math.pi * y / p.Ly + ph[1])[None, :, None]
        Z = (2 * math.pi * z / p.Lz + ph[2])[:, None, None]
        u = torch.sin(X) * torch.cos(Y) * torch.cos(Z) * one
        v = -torch.cos(X) * torch.sin(Y) * torch.cos(Z) * one
        w = 0 * one
        pr = Rgas + (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2.0) / 16.0 * one
        r = one
    elif flow == "channel":   # laminar profile and uniform noise on the velocities
        h = 0.5 * p.Lx
        u, v, w = (_noise(shape, seed * 8 + q, 0.1) for q in range(3))
        w = w + (1.5 * (1.0 - ((x - h) / h) ** 2))[None, None, :]
        r, pr = one, Rgas * one
    else:                  # boundary layer: the reference fields and smooth disturbances
        _, _, r2, u2, w2, e2 = (torch.tensor(a, device=_dev()) for a in _bl_refs(p))
        ph = np.random.default_rng(seed).uniform(0.0, 2 * math.pi, size=6)
        X, Y, Z = (2 * math.pi * x / p.Lx)[None, None, :], (2 * math.pi * y / p.Ly)[None, :, None], (2 * math.pi * z / p.Lz)[:, None, None]
        env = (1.0 - torch.exp(-x))[None, None, :]
        r = r2[:, None, :] * (1.0 + 0.002 * torch.cos(Y + ph[0]) * torch.cos(2 * Z + ph[1]) * env)
        u = u2[:, None, :] + 0.004 * env * torch.cos(Y + ph[2]) * torch.sin(3 * Z + ph[3]) * torch.sin(X)
        v = 0.004 * env * torch.sin(Y + ph[4]) * torch.cos(2 * Z + ph[5]) * one
        w = w2[:, None, :] * one
        pr = Rgas * one
    r, u, v, w = (a * one for a in (r, u, v, w))
    if developed and flow != "bl":
        r = r * (1.0 + 0.02 * torch.sin(2 * math.pi * x / p.Lx)[None, None, :] * torch.cos(4 * math.pi * y / p.Ly)[None, :, None])
        u, v, w = (a + _noise(shape, seed * 8 + 4 + q, 0.02) for q, a in enumerate((u, v, w)))
    e = pr / (p.gam - 1.0) + 0.5 * r * (u * u + v * v + w * w)
    return [r, u, v, w, e]


def _pinned(tensors):
    """Page-locked host arrays of the given device tensors, as numpy."""
    out = []
    for t in tensors:
        h = torch.empty(t.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
        h.copy_(t)
        out.append(h.numpy())
    return out


# ---------------------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        b = Batch(precision=PREC[case["prec"]])
        ids = [b.add(p, [f.cpu().numpy() for f in _fields(p, s, "tgv")], max_steps=4096)
               for p, s in _ensemble(case, seed)]
        return dict(kind=kind, batch=b, ids=ids, steps=case["steps"])
    if kind == "serve":
        reqs = [(p, [f.cpu().numpy() for f in _fields(p, s, "tgv" if p.periodic_x else "channel")])
                for p, s in _ensemble(case, seed)]
        return dict(kind=kind, server=Server(precision=PREC[case["prec"]]), requests=reqs, steps=case["steps"])
    p = _params(case)
    fields = _pinned(_fields(p, seed, case["flow"], kind != "run"))
    s = Solver(p)
    if case["flow"] == "bl":
        s.set_sponge(*_bl_refs(p))
    st = dict(kind=kind, solver=s, fields=fields)
    if kind == "run":
        st.update(out=_pinned([torch.zeros(p.shape, dtype=torch.float64)] * 5), steps=case["steps"],
                  dpdz=p.dpdz_init if p.forcing else 0.0)
    else:
        s.copy_field_in(*fields)
    return st


def run(st):
    kind = st["kind"]
    if kind == "batch":
        b = st["batch"]
        b.step(st["steps"])
        return [b.fields(i) for i in st["ids"]]
    if kind == "serve":
        srv = st["server"]
        rids = [srv.submit(p, f, st["steps"]) for p, f in st["requests"]]
        return [srv.wait(r) for r in rids]
    s = st["solver"]
    if kind == "rhs":
        return s.calc_rhs()
    if kind == "stats":
        return [s.plane_stats(), s.friction_reynolds(), s.dissipation()]
    s.copy_field_in(*st["fields"])
    s.set_scalars(0.0, st["dpdz"], 0.0)
    logs = s.run(st["steps"])
    return [s.copy_field_out(st["out"]), logs["par1"], logs["par2"], logs["time"]]


def work(case):
    """Per pass: the state and the Runge-Kutta register read and written once per stage (160
    bytes a point), the host fields once each way; flops of the split-form RHS, the state
    recovery and the stage update as the roofline counts them."""
    kind = case["kind"]
    if kind in ("batch", "serve"):
        n = sum(p.npoints for p, _ in _ensemble(case, 0))
        return dict(bytes=n * (480.0 * case["steps"] + (80.0 if kind == "serve" else 40.0)),
                    flops=n * 3.0 * case["steps"] * stage_flops(4, 4))
    n = float(case["mx"] * case["my"] * case["mz"])
    if kind == "rhs":
        return dict(bytes=n * 80.0, flops=n * stage_flops(case["S"], case["V"]))
    if kind == "stats":   # the fields once; gradients and dissipation, sums and squared deviations
        return dict(bytes=n * 40.0, flops=n * (9.0 * (3 * case["V"] + 1) + 80.0))
    ns = 4 if case["scheme"] == "rk4" else 3
    return dict(bytes=n * (80.0 + ns * STAGE_BYTES * case["steps"]),
                flops=n * ns * case["steps"] * stage_flops(case["S"], case["V"]))


# ---------------------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------------------
class _Ref:
    """The compressible Navier-Stokes right-hand side in split (Kennedy-Gruber) form, its
    boundary images, time step and Runge-Kutta schemes, field by field in torch."""

    def __init__(self, p, sponge=None):
        self.p = p
        T = lambda a: torch.tensor(np.asarray(a), dtype=torch.float64, device=_dev())  # noqa: E731
        x, xp, xpp, y, z = _grid(p)
        V = p.stencil_visc
        dx = (p.Lx / p.mx) if p.nonuniform_x else x[1] - x[0]
        self.inv = [1.0 / dx, 1.0 / (y[1] - y[0]), 1.0 / (z[1] - z[0])]
        self.c1S, _ = _weights(p.stencil_size)
        self.c1V, self.c2V = _weights(V)
        self.x = x
        self.xp0 = float(xp[0])
        self.xp, self.xpp = T(xp), T(xpp)
        dxv = np.empty(p.mx)
        dxv[0] = (x[1] + x[0]) / 2
        dxv[1:-1] = (x[2:] - x[:-2]) / 2
        dxv[-1] = p.Lx - (x[-1] + x[-2]) / 2
        self.dxv = T(dxv)
        self.wvol = self.dxv / self.inv[1] / self.inv[2]
        self.Ec = (p.gam - 1.0) * p.Ma * p.Ma
        self.Rgas = 1.0 / (p.gam * p.Ma * p.Ma)
        self.time, self.dt, self.dpdz = 0.0, 0.0, (p.dpdz_init if p.forcing else 0.0)
        self.sponge = None
        if sponge is not None:
            sx, sz, r, u, w, e = (T(a) for a in sponge)
            self.sponge = ((sx[None, :] + sz[:, None])[:, None, :],
                           [a[:, None, :] for a in (r, r * u, 0 * r, r * w, e)])

    def derived(self, q):
        p = self.p
        r, u, v, w, e = q
        T = (p.gam - 1.0) / self.Rgas * (e / r - 0.5 * (u * u + v * v + w * w))
        pr = r * self.Rgas * T
        return T, pr, (e + pr) / r, self.visc(T)

    def visc(self, T):
        return (T if self.p.viscexp == 1.0 else T ** self.p.viscexp) / self.p.Re

    # fields extended by G images on both sides along one axis (torch dim 2 - d)
    def _cat(self, f, d, lo, hi):
        return torch.cat([lo, f, hi], dim=2 - d)

    def _part(self, f, d, a, n):
        return f.narrow(2 - d, a, n)

    def _per(self, f, d):
        G, n = self.p.stencil_size, f.shape[2 - d]
        return self._cat(f, d, self._part(f, d, n - G, G), self._part(f, d, 0, G))

    def _mirror(self, f, d):
        G, n = self.p.stencil_size, f.shape[2 - d]
        return self._part(f, d, 0, G).flip(2 - d), self._part(f, d, n - G, G).flip(2 - d)

    def _extrap(self, f, d, high):
        G, n = self.p.stencil_size, f.shape[2 - d]
        if high:
            return 2 * self._part(f, d, n - 1, 1) - self._part(f, d, n - 1 - G, G).flip(2 - d)
        return 2 * self._part(f, d, 0, 1) - self._part(f, d, 1, G).flip(2 - d)

    def ext_state(self, F, d):
        """rho, u, v, w, T, p, H, mu extended along d."""
        p = self.p
        if d == 1 or (d == 2 and not p.boundary_layer) or (d == 0 and p.periodic_x):
            return [self._per(f, d) for f in F]
        if d == 2:
            return [self._cat(f, d, self._extrap(f, d, 0), self._extrap(f, d, 1)) for f in F]
        _, u, v, w, T, pr, _, _ = F
        sides = []
        for high in (0, 1):
            if p.boundary_layer and high:
                gu, gv, gw, gp, gT = (self._extrap(f, 0, 1) for f in (u, v, w, pr, T))
            else:
                gu, gv, gw, gp, gT = (self._mirror(f, 0)[high] for f in (u, v, w, pr, T))
                gu, gv, gw = -gu, -gv, -gw
                if not p.boundary_layer:
                    gT = 2.0 * (p.twall_top if high else p.twall_bot) - gT
                elif p.perturbed:
                    gu = self._perturb(gu)
            sides.append((gp / (self.Rgas * gT), gu, gv, gw, gT, gp,
                          gT * (self.Rgas * p.gam / (p.gam - 1.0)) + 0.5 * (gu * gu + gv * gv + gw * gw), self.visc(gT)))
        return [self._cat(f, 0, lo, hi) for f, lo, hi in zip(F, *sides)]

    def _perturb(self, gu):
        p = self.p
        k = np.arange(p.mz)
        st, en = p.pert_kc - p.pert_lp // 2, p.pert_kc + p.pert_lp // 2
        inside = (k >= st) & (k <= en)
        left = k < p.pert_kc
        ksi = np.where(left, (k - st) / (p.pert_kc - st), (en - k) / (en - p.pert_kc))
        g = 15.1875 * ksi ** 5 - 35.4375 * ksi ** 4 + 20.25 * ksi ** 3
        kap = np.where(left, 1.0, -1.0)
        y = np.arange(p.my) / self.inv[1]
        val = (p.pert_amp1 * math.sin(p.Re * p.pert_omega1_per_re * self.time)
               + p.pert_amp2 * math.sin(p.pert_omega2 * self.time) * np.cos(y / (p.Ly / (2 * math.pi)))[None, :]) * (kap * g)[:, None]
        val = torch.tensor(val, device=gu.device)[:, :, None]
        return torch.where(torch.tensor(inside, device=gu.device)[:, None, None], val.expand_as(gu), gu)

    def ext_theta(self, f, d):
        p = self.p
        if d == 1 or (d == 2 and not p.boundary_layer) or (d == 0 and p.periodic_x):
            return self._per(f, d)
        if d == 2:
            return self._cat(f, d, self._extrap(f, d, 0), self._extrap(f, d, 1))
        lo, hi = self._mirror(f, 0)
        return self._cat(f, 0, lo, self._extrap(f, 0, 1) if p.boundary_layer else hi)

    def at(self, E, d, l):
        G = self.p.stencil_size
        return E.narrow(2 - d, G + l, E.shape[2 - d] - 2 * G)

    def d1(self, E, d, c):
        s = sum(c[k] * (self.at(E, d, k) - self.at(E, d, -k)) for k in range(1, len(c))) * self.inv[d]
        return s * self.xp if d == 0 and self.p.nonuniform_x else s

    def d2(self, E, d):
        c = self.c2V
        s = (c[0] * self.at(E, d, 0) + sum(c[k] * (self.at(E, d, k) + self.at(E, d, -k)) for k in range(1, len(c)))) * self.inv[d] ** 2
        if d == 0 and self.p.nonuniform_x:
            f1 = sum(self.c1V[k] * (self.at(E, d, k) - self.at(E, d, -k)) for k in range(1, len(self.c1V))) * self.inv[0]
            return s * self.xp ** 2 - f1 * self.xpp * self.xp ** 3
        return s

    def gradients(self, X):
        return [[self.d1(X[d][1 + c], d, self.c1V) for c in range(3)] for d in range(3)]

    def rhs(self, q):
        p = self.p
        T, pr, H, mu = self.derived(q)
        F = [q[0], q[1], q[2], q[3], T, pr, H, mu]
        X = [self.ext_state(F, d) for d in range(3)]
        G = self.gradients(X)
        th = G[0][0] + G[1][1] + G[2][2]
        acc = [0.0] * 5
        W, L, cond, diss, LT = [0.0] * 3, [0.0] * 3, 0.0, 0.0, 0.0
        for d in range(3):
            r, u, v, w, t, pe, h, m = X[d]
            gn = X[d][1 + d]
            xs = self.xp if d == 0 and p.nonuniform_x else 1.0
            for a in range(1, len(self.c1S)):
                c = self.c1S[a] * self.inv[d] * xs
                qm = (self.at(r, d, -a) + q[0]) * (self.at(gn, d, -a) + q[1 + d])
                qp = (self.at(r, d, a) + q[0]) * (self.at(gn, d, a) + q[1 + d])
                acc[0] = acc[0] + 0.5 * c * (qm - qp)
                for n, (E, f0) in enumerate(((u, q[1]), (v, q[2]), (w, q[3]), (h, H)), 1):
                    acc[n] = acc[n] + 0.25 * c * (qm * (self.at(E, d, -a) + f0) - qp * (self.at(E, d, a) + f0))
            acc[1 + d] = acc[1 + d] - self.d1(pe, d, self.c1S)
            dm, dT, dth = self.d1(m, d, self.c1V), self.d1(t, d, self.c1V), self.d1(self.ext_theta(th, d), d, self.c1V)
            for c in range(3):
                tau = G[d][c] + G[c][d] - (2.0 / 3.0 * th if c == d else 0.0)
                W[c] = W[c] + tau * dm
                L[c] = L[c] + self.d2(X[d][1 + c], d)
                g = G[d][c]
                if d == 1 and c == 2 and p.quirk_dissipation_y:
                    g = G[2][1]   # the reference's tau_yz dv/dz in the y sum
                diss = diss + tau * g
            W[d] = W[d] + mu / 3.0 * dth
            cond = cond + dT * dm
            LT = LT + self.d2(t, d)
        cond = cond + mu * LT
        for c in range(3):
            W[c] = W[c] + mu * L[c]
            acc[1 + c] = acc[1 + c] + W[c]
        acc[4] = acc[4] + mu * diss + cond / (p.Pr * self.Ec) + q[1] * W[0] + q[2] * W[1] + q[3] * W[2]
        acc[3] = acc[3] + self.dpdz
        acc[4] = acc[4] + self.dpdz * q[3]
        if self.sponge is not None:
            s, ref = self.sponge
            for n, f in enumerate((q[0], q[0] * q[1], q[0] * q[2], q[0] * q[3], q[4])):
                acc[n] = acc[n] + s * (ref[n] - f)
        return acc

    def checks(self, q):
        """dt (and the body force) and the bulk diagnostics of the state."""
        p = self.p
        r, u, v, w, e = q
        k2 = u * u + v * v + w * w
        c = torch.sqrt(p.gam * (p.gam - 1.0) * (e / r - 0.5 * k2))
        conv = torch.maximum((u.abs() + c) / self.dxv, torch.maximum((v.abs() + c) * self.inv[1], (w.abs() + c) * self.inv[2]))
        mu = self.derived(q)[3]
        vis = torch.maximum(mu / self.dxv ** 2, mu * max(self.inv[1], self.inv[2]) ** 2)
        self.dt = min(1e5, p.cfl / float(torch.maximum(conv, vis).max()))
        vol = p.Lx * p.Ly * p.Lz
        if p.forcing:
            bulk = float((r * w * self.wvol).sum() / (r * self.wvol).sum())
            self.dpdz = 0.99 * self.dpdz - 0.5 * (bulk - 1.0)
            return bulk, float((e * self.wvol).sum())
        return float((k2 * self.wvol).sum()) / vol, 0.5 * float((r * k2 * self.wvol).sum()) / vol

    def advance(self, q, steps):
        """`steps` steps (fewer than the check period) from a fresh start: state and logs."""
        par = self.checks(q)
        C = [q[0], q[0] * q[1], q[0] * q[2], q[0] * q[3], q[4]]
        prim = lambda c: [c[0], c[1] / c[0], c[2] / c[0], c[3] / c[0], c[4]]  # noqa: E731
        times = []
        dt = self.dt
        for _ in range(steps):
            self.time += dt
            if self.p.scheme == RK3_LOWSTORAGE:
                prev = None
                for a, b in ((0.0, 8 / 15), (-17 / 60, 5 / 12), (-5 / 12, 3 / 4)):
                    R = self.rhs(prim(C))
                    C = [c + dt * (b * x + (a * y if prev is not None else 0.0)) for c, x, y in zip(C, R, prev or R)]
                    prev = R
            elif self.p.scheme == RK3_CLASSIC:
                k1 = self.rhs(prim(C))
                k2 = self.rhs(prim([c + 0.5 * dt * a for c, a in zip(C, k1)]))
                k3 = self.rhs(prim([c + dt * (2 * b - a) for c, a, b in zip(C, k1, k2)]))
                C = [c + dt * (a + 4 * b + x) / 6 for c, a, b, x in zip(C, k1, k2, k3)]
            else:
                k1 = self.rhs(prim(C))
                k2 = self.rhs(prim([c + 0.5 * dt * a for c, a in zip(C, k1)]))
                k3 = self.rhs(prim([c + 0.5 * dt * a for c, a in zip(C, k2)]))
                k4 = self.rhs(prim([c + dt * a for c, a in zip(C, k3)]))
                C = [c + dt / 6 * (a + 2 * b + 2 * x + y) for c, a, b, x, y in zip(C, k1, k2, k3, k4)]
            times.append(self.time)
        logs = [np.full(steps, np.nan), np.full(steps, np.nan), np.array(times)]
        logs[0][0], logs[1][0] = par
        return prim(C), logs

    def stats(self, q):
        p = self.p
        r, u, v, w, e = q
        n = p.my * p.mz
        m = [f.sum((0, 1)) / n for f in (r, r * u, r * v, r * w, e)]
        m = [m[0], m[1] / m[0], m[2] / m[0], m[3] / m[0], m[4]]
        dev = [((f - a) ** 2).sum((0, 1)) / n for f, a in zip(q, m)]
        prof = torch.stack([torch.tensor(self.x, device=r.device)] + m + dev)
        d = sum(self.c1S[k] * (w[:, :, k] - w[:, :, k - 1]) for k in range(1, len(self.c1S))) * self.inv[0] * self.xp0
        muw = 1.0 / p.Re
        ret = (torch.sqrt(muw * d.abs() / r[:, :, 0]) * r[:, :, 0] / muw).sum() / n
        T, pr, H, mu = self.derived(q)
        X = [self.ext_state([r, u, v, w, T, pr, H, mu], k) for k in range(3)]
        G = self.gradients(X)
        th = G[0][0] + G[1][1] + G[2][2]
        s = sum((G[a][b] + G[b][a] - (2.0 / 3.0 * th if a == b else 0.0)) * G[a][b] for a in range(3) for b in range(3))
        om = (G[1][2] - G[2][1]) ** 2 + (G[2][0] - G[0][2]) ** 2 + (G[0][1] - G[1][0]) ** 2
        vol = p.Lx * p.Ly * p.Lz
        return [prof.cpu().numpy(), float(ret), dict(eps=float((mu * s * self.wvol).sum()) / vol,
                                                     enstrophy=float((om * self.wvol).sum()) / vol)]


def _host(fields):
    return [(f + torch.zeros_like(fields[0])).cpu().numpy() if isinstance(f, torch.Tensor) else f for f in fields]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        out = []
        for p, s in _ensemble(case, seed):
            q, _ = _Ref(p).advance(_fields(p, s, "tgv" if p.periodic_x else "channel"), case["steps"])
            out.append(_host(q))
        return out
    p = _params(case)
    q = _fields(p, seed, case["flow"], kind != "run")
    ref = _Ref(p, _bl_refs(p) if case["flow"] == "bl" else None)
    if kind == "rhs":
        return _host(ref.rhs(q))
    if kind == "stats":
        return ref.stats(q)
    q, logs = ref.advance(q, case["steps"])
    return [_host(q)] + logs
