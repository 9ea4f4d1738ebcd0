"""Workloads of the WENO-GKS library, as a user's program runs them.

Every case goes through the public binding (gks_b200.Solver).  The kinds:

  step       the resident field advanced `steps` steps (gks_step): the time
             loop between two outputs
  ensemble   the same for a batch of independent fields of several sizes
  loop       the reference's Evolve loop, `steps` times one step and one
             statistics line (PrintStats every step)
  stats      one statistics call on the resident field
  particles  the driver's loop with particles, `steps` times: spline
             properties at every particle, their statistics, the particles'
             move, the field's step; then the particle records
  evolve     the reference's per-step call evolve(W, dev, dt) on pinned host
             memory, `steps` times

Inputs: decaying isotropic turbulence (random-phase solenoidal velocity with
the spectrum n^4 exp(-2 n^2 / k0^2), k0 = 4, scaled to the turbulent Mach
number) with density and pressure fluctuations of the order Mt^2, made on the
GPU from the seed.  `exact` restates the scheme in plain torch, in the
reference's own form (1-D moment tables contracted per moment vector).
"""

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gkm-dns_b200"))

import gks_b200 as gks  # noqa: E402

GAM, GAS_R, RHO0, K0, CFL = 1.4, 287.0, 1.0, 4.0, 0.5
P0 = RHO0 / GAM  # sound speed 1
T0 = P0 / (GAS_R * RHO0)
KDOF = 2  # int((5 - 3 gam) / (gam - 1))
VISC_EXP = 0.76
EXACT_CELLS = 130**3  # most cells x steps the plain torch restatement takes on

PRECISION = {"fp64": gks.FP64, "mixed": gks.MIXED}


def _case(kind, nc, precision="fp64", steps=1, mach=0.5, re=100.0, **more):
    return {"kind": kind, "nc": nc, "precision": precision, "steps": steps, "mach": mach, "re": re, **more}


def listed():
    def named(name, *a, **k):
        return {"name": name, **_case(*a, **k)}

    return [
        # small field, ten steps between two outputs: latency and launches
        named("step-32", "step", 32, steps=10, mach=0.3, re=72.0),
        # odd size, the options of the reference's GPU semantics (energy reconstructed
        # directly, Prandtl factor 1) with the rotated z sweep and the power-law viscosity
        named("step-75-gpu-semantics", "step", 75, steps=2, direct=True, fixz=True, power=True),
        # ordinary field
        named("step-128-mixed", "step", 128, precision="mixed", mach=0.3, re=72.0),
        # the benchmark's field, both precisions
        named("step-256", "step", 256),
        named("step-256-mixed", "step", 256, precision="mixed"),
        # the largest field the configurations name
        named("step-512-mixed", "step", 512, precision="mixed", mach=0.4, re=150.0),
        # ensemble of 96 fields, 32 of each size
        named("ensemble-96", "ensemble", 64, sizes="32,48,64", each=32),
        # the driver's default loop: statistics every step
        named("loop-130", "loop", 130, steps=2, mach=0.3, re=72.0),
        # statistics of the benchmark's field alone
        named("stats-256", "stats", 256),
        # host call on a small field: latency, launches and copies
        named("evolve-48", "evolve", 48, mach=0.3, re=72.0),
        # host call on the benchmark's field: PCIe both ways
        named("evolve-256", "evolve", 256),
        # driver loop with 2^20 particles, ten steps between two outputs of the records
        named("particles-256", "particles", 256, steps=10, particles=1 << 20),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "step", "ensemble", "loop", "stats", "evolve", "particles"])
    common = {"precision": rng.choice(["fp64", "mixed"]), "mach": round(rng.uniform(0.2, 0.6), 3),
              "re": round(rng.uniform(40.0, 160.0), 1)}
    if kind == "step":
        nc = size(12, 300)
        return _case(kind, nc, steps=rng.randint(1, 10) if nc < 100 else 1, direct=rng.random() < 0.25,
                     fixz=rng.random() < 0.25, power=rng.random() < 0.25, **common)
    if kind == "ensemble":
        sizes = sorted(size(12, 72) for _ in range(3))
        return _case(kind, sizes[-1], sizes=",".join(map(str, sizes)), each=rng.randint(2, 16), **common)
    if kind == "loop":
        return _case(kind, size(16, 200), steps=rng.randint(1, 4), **common)
    if kind == "stats":
        return _case(kind, size(16, 300), **common)
    if kind == "evolve":
        return _case(kind, size(16, 200), **common)
    return _case(kind, size(16, 160), steps=rng.randint(1, 4), particles=size(1000, 1 << 20), **common)


def _sizes(case):
    if case["kind"] == "ensemble":
        return [int(s) for s in case["sizes"].split(",") for _ in range(case["each"])]
    return [case["nc"]]


# --------------------------------------------------------------------------- inputs
def _constants(case):
    urms = case["mach"] / math.sqrt(3.0)
    lam = 2.0 / K0
    return {"mu0": RHO0 * urms * lam / case["re"], "t0": lam / urms, "pr": 1.0 if case.get("direct") else 1.0 / 0.7}


def _phys(case, nc):
    c = _constants(case)
    return gks.Phys(nc=nc, K=KDOF, visc_law=gks.VISC_POWER if case.get("power") else gks.VISC_SUTHERLAND, reserved=0,
                    gam=GAM, gas_r=GAS_R, T0=T0, mu0=c["mu0"], visc_exp=VISC_EXP, pr_factor=c["pr"], p0=P0, den0=RHO0,
                    Mt=case["mach"], t0=c["t0"])


def _flags(case):
    return (gks.DIRECT_ENERGY if case.get("direct") else 0) | (gks.FIX_ZSWEEP if case.get("fixz") else 0)


def _field(nc, mach, gen):
    """The five conservative fields on the interior, (5, nc, nc, nc) = [q, y, x, z]."""
    kf = torch.fft.fftfreq(nc, d=1.0 / nc, device="cuda", dtype=torch.float64)
    kz = torch.arange(nc // 2 + 1, device="cuda", dtype=torch.float64)
    k2 = kf[:, None, None] ** 2 + kf[None, :, None] ** 2 + kz[None, None, :] ** 2
    shape = torch.exp(-k2 / (K0 * K0)) * k2  # amplitude of E(n) = n^4 exp(-2 n^2 / k0^2) per mode
    k2[0, 0, 0] = 1.0

    def mode():
        x = torch.rand((nc, nc, nc), generator=gen, device="cuda", dtype=torch.float64)
        return torch.fft.rfftn(x - 0.5) * shape

    W = torch.empty((5, nc, nc, nc), device="cuda", dtype=torch.float64)
    u = [mode(), mode(), mode()]  # components along x, y, z
    wave = [kf[None, :, None], kf[:, None, None], kz[None, None, :]]
    div = sum(a * k for a, k in zip(u, wave)) / k2
    for q in range(3):
        W[1 + q] = torch.fft.irfftn(u[q] - div * wave[q], s=(nc, nc, nc))
    del u, div
    W[1:4] *= mach / W[1:4].square().sum(0).mean().sqrt()
    fl = torch.fft.irfftn(mode() / k2.sqrt(), s=(nc, nc, nc))
    fl *= mach * mach / fl.abs().max()
    p = P0 * (1.0 + 0.5 * fl)
    fl = torch.fft.irfftn(mode() / k2.sqrt(), s=(nc, nc, nc))
    fl *= mach * mach / fl.abs().max()
    W[0] = RHO0 * (p / P0) ** (1.0 / GAM) * (1.0 + 0.25 * fl)
    W[4] = p / (GAM - 1.0) + 0.5 * W[0] * W[1:4].square().sum(0)
    W[1:4] *= W[0]
    return W


def _fields(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    for nc in _sizes(case):
        yield _field(nc, case["mach"], gen)


def _positions(case, seed):
    return np.random.default_rng(seed).random((3, case["particles"])) * (2.0 * math.pi)


class _Array:
    """A field's resident array as torch sees it; keeps the solver alive."""

    def __init__(self, solver, ptr, nc):
        self.solver = solver
        self.__cuda_array_interface__ = {"shape": (nc, nc, nc), "typestr": "<f8", "data": (ptr, False), "version": 3}


def _resident(state):
    """The fields' resident arrays, as torch tensors (the state itself, no copy)."""
    s, views = state["solver"], state["views"]
    out = []
    for f, p in enumerate(s.phys):
        for ptr in s.device_fields(f):
            if ptr not in views:
                views[ptr] = torch.as_tensor(_Array(s, ptr, p.nc), device="cuda")
            out.append(views[ptr])
    return out


def prepare(case, seed):
    sizes = _sizes(case)
    s = gks.Solver([_phys(case, nc) for nc in sizes], PRECISION[case["precision"]], _flags(case))
    state = {"case": case, "solver": s, "views": {}}
    if case["kind"] == "evolve":
        W = next(_fields(case, seed)).cpu().numpy()
        host = torch.empty(s.host_shape(), dtype=torch.float64, pin_memory=True)
        host.numpy()[...] = np.pad(W, ((0, 0), (3, 3), (3, 3), (3, 3)), mode="wrap")
        state["host"] = host
        s.set_dt(_dt(torch.from_numpy(W), case))
        return state
    arrays = _resident(state)
    for f, W in enumerate(_fields(case, seed)):
        for q in range(5):
            arrays[5 * f + q].copy_(W[q])
        del W
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    state["dt"] = [s.timestep(CFL, f) for f in range(len(sizes))]
    if case["kind"] == "particles":
        s.particles_locate(*_positions(case, seed))
    return state


def run(state):
    case, s = state["case"], state["solver"]
    kind = case["kind"]
    if kind == "evolve":
        W = state["host"].numpy()
        for _ in range(case["steps"]):
            s.evolve(W)
        return state["host"]
    if kind == "stats":
        return s.stats_array()
    if kind == "loop":
        lines = []
        for _ in range(case["steps"]):
            lines.append(s.stats_array())
            s.step(1)
        return {"lines": np.array(lines), "W": _resident(state)}
    if kind == "particles":
        lines = []
        for _ in range(case["steps"]):
            s.particles_props()
            lines.append(s.particles_stats())
            s.particles_track(state["dt"][0])
            s.step(1)
        return {"lines": np.array(lines), "records": s.particles_get(), "W": _resident(state)}
    s.step(case["steps"])
    if kind == "ensemble":
        s.sync()  # the gathering below runs on torch's stream
        arrays = _resident(state)
        return [torch.cat([a.reshape(-1) for a in arrays[q::5]]) for q in range(5)]
    return _resident(state)


def work(case):
    """Bytes: the state read and written once per step (and over PCIe once each
    way for the host call), the records once.  Flops: the scheme's per-cell
    count of one step (three interfaces of flux, 2300, and of reconstruction,
    700), of a statistics call and of the particles' splines."""
    n = sum(nc**3 for nc in _sizes(case))
    kind, steps = case["kind"], case["steps"]
    step = {"bytes": 80.0 * n, "flops": 9000.0 * n}
    stats = {"bytes": 40.0 * n, "flops": 250.0 * n}
    if kind == "stats":
        return stats
    w = {k: steps * v for k, v in step.items()}
    if kind == "loop":
        w = {k: v + steps * stats[k] for k, v in w.items()}
    elif kind == "evolve":
        w["bytes"] += steps * 80.0 * (case["nc"] + 6) ** 3
    elif kind == "particles":
        m = case["particles"]
        w["bytes"] += steps * (40.0 * n + 2 * 8.0 * gks.PREC_FIELDS * m) + 8.0 * gks.PREC_FIELDS * m
        w["flops"] += steps * (100.0 * n + 3600.0 * m)
    return w


# --------------------------------------------------------------------------- plain torch restatement
def _prim(W):
    den = W[0]
    u = [W[1] / den, W[2] / den, W[3] / den]
    p = (den * (GAM - 1)) * (W[4] / den - 0.5 * (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]))
    return den, u, p


def _dt(W, case):
    den, u, p = _prim(W)
    speed = (u[0] * u[0] + u[1] * u[1] + u[2] * u[2]).sqrt() + (GAM * p / den).sqrt()
    return CFL * (2.0 * math.pi / W.shape[-1]) / float(speed.max())


def _viscosity(case, T):
    mu0 = _constants(case)["mu0"]
    if case.get("power"):
        return mu0 * (T / T0) ** VISC_EXP
    return mu0 * (T / T0) ** 1.5 * (T0 + 110.4) / (T + 110.4)


def _weno(s):
    """WENO-SYMOO left and right interface values from six shifted arrays."""

    def side(a, b, c, d, e, f):
        p = (a / 3 - 7 * b / 6 + 11 * c / 6, -b / 6 + 5 * c / 6 + d / 3, c / 3 + 5 * d / 6 - e / 6,
             11 * d / 6 - 7 * e / 6 + f / 3)
        i0 = 13 * (a - 2 * b + c) ** 2 / 12 + (a - 4 * b + 3 * c) ** 2 / 4
        i1 = 13 * (b - 2 * c + d) ** 2 / 12 + (d - b) ** 2 / 4
        i2 = 13 * (c - 2 * d + e) ** 2 / 12 + (3 * c - 4 * d + e) ** 2 / 4
        i3 = 13 * (d - 2 * e + f) ** 2 / 12 + (5 * d - 8 * e + 3 * f) ** 2 / 4
        i3 = torch.maximum(torch.maximum(torch.maximum(i0, i1), i2), i3)
        al = [g / (1e-10 + i) for g, i in zip((0.05, 0.45, 0.45, 0.05), (i0, i1, i2, i3))]
        return sum(x * y for x, y in zip(al, p)) / (al[0] + al[1] + al[2] + al[3])

    return side(*s), side(*s[::-1])


def _reconstruct(W, dim, direct):
    """Left and right states at the interface above each cell along `dim`."""

    def pair(a):
        return _weno([torch.roll(a, 2 - d, dim) for d in range(6)])

    wl, wr = zip(*(pair(W[q]) for q in range(4)))
    wl, wr = list(wl), list(wr)
    if direct:
        el, er = pair(W[4])
    else:
        _, _, p = _prim(W)
        tl, tr = pair(p / (GAS_R * W[0]))
        el, er = (w[0] * GAS_R * t / (GAM - 1.0) + 0.5 * (w[1] ** 2 + w[2] ** 2 + w[3] ** 2) / w[0]
                  for w, t in ((wl, tl), (wr, tr)))
    return wl + [el], wr + [er]


class _Maxwellian:
    def __init__(self, W):
        self.den, self.U, p = _prim(W)
        self.lam = 0.5 * self.den / p
        s = 0.5 / self.lam
        self.s = s
        self.full = [self._table(u, torch.ones_like(u), u, 7) for u in self.U]
        self.e2 = KDOF * s
        self.e4 = (KDOF * KDOF + 2 * KDOF) * s * s

    def _table(self, u, m0, m1, n):
        t = [m0, m1]
        for k in range(2, n):
            t.append(u * t[-1] + (k - 1) * self.s * t[-2])
        return t

    def half(self, sign):
        u, root = self.U[0], self.lam.sqrt()
        m0 = 0.5 * torch.erfc(-sign * root * u)
        return self._table(u, m0, u * m0 + sign * 0.5 * torch.exp(-self.lam * u * u) / (math.sqrt(math.pi) * root), 7)

    def moment(self, X, k, lm, a):
        """<psi u^k v^l w^m (a . psi)>, or <psi u^k> without a."""
        Y, Z, e2, e4 = self.full[1], self.full[2], self.e2, self.e4
        l, m = lm
        cache = {}

        def t(i, j, n):
            if (i, j, n) not in cache:
                cache[i, j, n] = X[k + i] * Y[l + j] * Z[m + n]
            return cache[i, j, n]

        def energy(i, j, n):
            return 0.5 * (t(i + 2, j, n) + t(i, j + 2, n) + t(i, j, n + 2) + t(i, j, n) * e2)

        unit = ((1, 0, 0), (0, 1, 0), (0, 0, 1))
        if a is None:
            return [t(0, 0, 0)] + [t(*d) for d in unit] + [energy(0, 0, 0)]
        v = [energy(0, 0, 0)] + [energy(*d) for d in unit]
        M = [sum((a[1 + i] * t(*d) for i, d in enumerate(unit)), a[0] * t(0, 0, 0) + a[4] * v[0])]
        for i, d in enumerate(unit):
            M.append(sum((a[1 + j] * t(*(x + y for x, y in zip(d, e))) for j, e in enumerate(unit)),
                         a[0] * t(*d) + a[4] * v[1 + i]))
        v4 = 0.25 * (t(4, 0, 0) + t(0, 4, 0) + t(0, 0, 4) + t(0, 0, 0) * e4 +
                     2 * (t(2, 2, 0) + t(2, 0, 2) + t(0, 2, 2)) + 2 * e2 * (t(2, 0, 0) + t(0, 2, 0) + t(0, 0, 2)))
        M.append(a[0] * v[0] + a[1] * v[1] + a[2] * v[2] + a[3] * v[3] + a[4] * v4)
        return M

    def slopes(self, b, pr):
        U, lam = self.U, self.lam
        q = U[0] * U[0] + U[1] * U[1] + U[2] * U[2] + (KDOF + 3) * self.s
        R = [b[1 + i] - U[i] * b[0] for i in range(3)]
        a4 = pr * (2 * b[4] - b[0] * q - 2 * (U[0] * R[0] + U[1] * R[1] + U[2] * R[2])) * (4 * lam * lam) / (KDOF + 3)
        a = [2 * lam * R[i] - U[i] * a4 for i in range(3)]
        a0 = b[0] - a[0] * U[0] - a[1] * U[1] - a[2] * U[2] - 0.5 * a4 * q
        return [a0] + a + [a4]


def _add(*vs):
    return [sum(x[1:], x[0]) for x in zip(*vs)]


def _mul(c, v):
    return [c * x for x in v]


def _flux(WL, WR, Wl, Wr, Dl, Dr, tau, dt, dx, pr):
    """Time-integrated BGK-NS flux; states rotated so that component 1 is normal."""
    l, r = _Maxwellian(Wl), _Maxwellian(Wr)
    Xl, Xr = l.half(1), r.half(-1)
    none, ty, tz = (0, 0), (1, 0), (0, 1)
    W0 = _add(_mul(l.den, l.moment(Xl, 0, none, None)), _mul(r.den, r.moment(Xr, 0, none, None)))
    e = _Maxwellian(W0)
    al = [l.slopes([x / l.den for x in d], pr) for d in Dl]
    ar = [r.slopes([x / r.den for x in d], pr) for d in Dr]
    exl = e.slopes([2 * (a - b) / (e.den * dx) for a, b in zip(W0, WL)], pr)
    exr = e.slopes([2 * (b - a) / (e.den * dx) for a, b in zip(W0, WR)], pr)
    ey = e.slopes(_add(l.moment(Xl, 0, none, al[1]), r.moment(Xr, 0, none, ar[1])), pr)
    ez = e.slopes(_add(l.moment(Xl, 0, none, al[2]), r.moment(Xr, 0, none, ar[2])), pr)

    def convect(g, X, k, a):
        return _add(g.moment(X, k + 1, none, a[0]), g.moment(X, k, ty, a[1]), g.moment(X, k, tz, a[2]))

    Al = l.slopes(_mul(-1.0, convect(l, l.full[0], 0, al)), pr)
    Ar = r.slopes(_mul(-1.0, convect(r, r.full[0], 0, ar)), pr)
    w = (l.den / l.lam - r.den / r.lam).abs() / (l.den / l.lam + r.den / r.lam).abs()
    tau = tau + dt * w
    ex = torch.exp(-dt / tau)
    om = -torch.expm1(-dt / tau)
    gm0 = dt - tau * om
    gm1, gm2, gm4 = -om / gm0, (-dt + 2 * tau * om - dt * ex) / gm0, (dt * ex - tau * om) / gm0
    gm3, gm5 = -gm1, -tau * gm1
    Xe = e.full[0]
    Xp, Xn = e.half(1), e.half(-1)

    def equilibrium(k):
        return _add(e.moment(Xp, k + 1, none, exl), e.moment(Xn, k + 1, none, exr), e.moment(Xe, k, ty, ey),
                    e.moment(Xe, k, tz, ez))

    cl, cr = _mul(l.den, convect(l, Xl, 0, al)), _mul(r.den, convect(r, Xr, 0, ar))
    cA = _add(_mul(l.den, l.moment(Xl, 0, none, Al)), _mul(r.den, r.moment(Xr, 0, none, Ar)))
    B = _add(_mul(gm1 * e.den, e.moment(Xe, 0, none, None)), _mul(gm2 * e.den, equilibrium(0)), _mul(gm3, W0),
             _mul(gm4 + gm5, _add(cl, cr)), _mul(gm5, cA))
    A = e.slopes([b / e.den for b in B], pr)
    P = tau * om
    Q = -tau * dt * ex + tau * tau * om
    p0 = dt - P
    p1, p2 = 0.5 * dt * dt - tau * p0, -tau * p0 + Q
    p4, p5 = -Q - tau * P, -tau * P
    f0 = _add(_mul(l.den, l.moment(Xl, 1, none, None)), _mul(r.den, r.moment(Xr, 1, none, None)))
    fx = _add(_mul(l.den, convect(l, Xl, 1, al)), _mul(r.den, convect(r, Xr, 1, ar)))
    fA = _add(_mul(l.den, l.moment(Xl, 1, none, Al)), _mul(r.den, r.moment(Xr, 1, none, Ar)))
    return _add(_mul(p0 * e.den, e.moment(Xe, 1, none, None)), _mul(p1 * e.den, e.moment(Xe, 1, none, A)),
                _mul(p2 * e.den, equilibrium(1)), _mul(P, f0), _mul(p4, fx), _mul(p5, fA))


def _rotate(v, slot):
    v = list(v)
    v[1], v[slot] = v[slot], v[1]
    return v


def _net_flux(W, case, dt, dx):
    """Sum over the three directions of F(cell) - F(cell - 1), arrays [y, x, z]."""
    pr = _constants(case)["pr"]
    den, _, p = _prim(W)
    tau = _viscosity(case, p / (GAS_R * den)) / p
    Y, X, Z = 0, 1, 2  # array dimensions
    # sweep dimension, dimension of the first and second transverse slope, momentum slot of the normal
    zt = (Y, X) if case.get("fixz") else (X, Y)
    total = None
    for dim, t1, t2, slot in ((X, Y, Z, 1), (Y, X, Z, 2), (Z, *zt, 3)):
        wl, wr = _reconstruct(W, dim, bool(case.get("direct")))
        wc = [W[q] for q in range(5)]
        wn = [torch.roll(x, -1, dim) for x in wc]

        def slopes(w, normal):
            side = [normal] + [[0.5 * (torch.roll(x, -1, t) - torch.roll(x, 1, t)) / dx for x in w] for t in (t1, t2)]
            return [_rotate(d, slot) for d in side]

        Dl = slopes(wl, [2 * (a - b) / dx for a, b in zip(wl, wc)])
        Dr = slopes(wr, [2 * (b - a) / dx for a, b in zip(wr, wn)])
        F = _rotate(_flux(_rotate(wc, slot), _rotate(wn, slot), _rotate(wl, slot), _rotate(wr, slot), Dl, Dr, tau, dt,
                          dx, pr), slot)
        d = torch.stack([f - torch.roll(f, 1, dim) for f in F])
        total = d if total is None else total + d
    return total


def _step(W, case, dt):
    n = W.shape[-1]
    dx = 2.0 * math.pi / n
    inner = max(8, (1 << 22) // (n * n))
    if inner + 8 >= n:
        return W - _net_flux(W, case, dt, dx) / dx
    out = torch.empty_like(W)
    for j in range(0, n, inner):  # blocks of planes with four more on either side, whose results are dropped
        m = min(inner, n - j)
        planes = torch.arange(j - 4, j + m + 4, device=W.device) % n
        out[:, j:j + m] = W[:, j:j + m] - _net_flux(W[:, planes], case, dt, dx)[:, 4:4 + m] / dx
    return out


def _pad(n):
    """Padded periodic line (three ghosts either side) of an interior line, as a matrix."""
    P = torch.zeros((n + 6, n), dtype=torch.float64, device="cuda")
    P[torch.arange(n + 6), torch.arange(-3, n + 3) % n] = 1.0
    return P


def _along(M, a, dim):
    return torch.movedim(torch.tensordot(M, a, dims=([1], [dim])), 0, dim)


def _stats(W, case):
    """PrintStats' quantities, velocity gradients from natural cubic splines through each padded line."""
    n = W.shape[-1]
    h = 2.0 * math.pi / n
    nt = n + 6
    A = torch.zeros((nt, nt), dtype=torch.float64, device="cuda")
    R = torch.zeros_like(A)
    i = torch.arange(1, nt - 1)
    A[i, i - 1], A[i, i], A[i, i + 1] = 1.0, 4.0, 1.0
    R[i, i + 1], R[i, i - 1] = 3.0 / h, -3.0 / h
    A[0, 0], A[0, 1], A[-1, -1], A[-1, -2] = 2.0, 1.0, 2.0, 1.0
    R[0, 0], R[0, 1], R[-1, -2], R[-1, -1] = -3.0 / h, 3.0 / h, -3.0 / h, 3.0 / h
    G = torch.linalg.solve(A, R @ _pad(n))[3:-3]
    den, u, p = _prim(W)
    T = p / (GAS_R * den)
    mu = _viscosity(case, T)
    g = [[_along(G, c, d) for d in (1, 0, 2)] for c in u]  # g[component][x, y, z]
    m = lambda x: float(x.mean())  # noqa: E731
    u2 = u[0] * u[0] + u[1] * u[1] + u[2] * u[2]
    diss = m(mu * sum(x * x for r in g for x in r))
    sij = m(g[0][0] ** 2 + g[1][1] ** 2 + g[2][2] ** 2 + 0.5 * ((g[0][1] + g[1][0]) ** 2 + (g[0][2] + g[2][0]) ** 2 +
                                                              (g[1][2] + g[2][1]) ** 2))
    d2 = [m(g[c][c] ** 2) for c in range(3)]
    skew = [m(g[c][c] ** 3) / d2[c] ** 1.5 for c in range(3)]
    kurt = [m(g[c][c] ** 4) / d2[c] ** 2 for c in range(3)]
    rms = lambda x: math.sqrt(m((x - x.mean()) ** 2))  # noqa: E731
    M = case["mach"]
    return np.array([m(den * u2), diss, *skew, *kurt, rms(p) / (GAM * P0 * M * M), rms(T) / ((GAM - 1) * T0 * M * M),
                     rms(1 / den) / (M * M / RHO0), sij, math.sqrt(m(u2)) / m((GAM * p / den).sqrt()), m(den)])


def _spline_matrix(nt):
    """Natural cubic B-spline coefficients (nt + 2) of nt nodal values, as a matrix."""
    A = torch.zeros((nt + 2, nt + 2), dtype=torch.float64, device="cuda")
    i = torch.arange(nt)
    A[i, i], A[i, i + 1], A[i, i + 2] = 1 / 6, 4 / 6, 1 / 6
    A[nt, 0], A[nt, 1], A[nt, 2] = 1.0, -2.0, 1.0
    A[nt + 1, -1], A[nt + 1, -2], A[nt + 1, -3] = 1.0, -2.0, 1.0
    rhs = torch.zeros((nt + 2, nt), dtype=torch.float64, device="cuda")
    rhs[i, i] = 1.0
    return torch.linalg.solve(A, rhs)


def _props(W, pos):
    """Values (5, n) and gradients (5, 3, n) of den, u, v, w, p at pos = (y, x, z)."""
    n = W.shape[-1]
    nt = n + 6
    h = 2.0 * math.pi / n
    C = _spline_matrix(nt) @ _pad(n)
    den, u, p = _prim(W)
    at, wt, dwt = [], [], []
    for x in pos:
        c = (x + 2.5 * h) / h
        i = c.floor().clamp(0, nt - 2)
        t = c - i
        at.append(i.long())
        wt.append(((1 - t) ** 3 / 6, (3 * t**3 - 6 * t**2 + 4) / 6, (-3 * t**3 + 3 * t**2 + 3 * t + 1) / 6, t**3 / 6))
        dwt.append((-0.5 * (1 - t) ** 2, 1.5 * t**2 - 2 * t, -1.5 * t**2 + t + 0.5, 0.5 * t**2))
    values, grads = [], []
    for f in (den, *u, p):
        c = f
        for d in range(3):
            c = _along(C, c, d)
        M = nt + 2
        c = c.reshape(-1)
        v, gy, gx, gz = 0.0, 0.0, 0.0, 0.0
        for a in range(4):
            for b in range(4):
                base = ((at[0] + a) * M + at[1] + b) * M + at[2]
                rows = [c[base + k] for k in range(4)]
                s = sum(w * r for w, r in zip(wt[2], rows))
                v = v + wt[0][a] * wt[1][b] * s
                gy = gy + dwt[0][a] * wt[1][b] * s
                gx = gx + wt[0][a] * dwt[1][b] * s
                gz = gz + wt[0][a] * wt[1][b] * sum(w * r for w, r in zip(dwt[2], rows))
        values.append(v)
        grads.append([gy / h, gx / h, gz / h])
    return values, grads


def _particle_line(values, grads):
    u, g = values[1:4], grads[1:4]  # g[component][y, x, z]
    m = lambda x: float(x.mean())  # noqa: E731
    sij = m(g[0][1] ** 2 + g[1][0] ** 2 + g[2][2] ** 2 + 0.5 * ((g[0][0] + g[1][1]) ** 2 + (g[0][2] + g[2][1]) ** 2 +
                                                              (g[2][0] + g[1][2]) ** 2))
    x2, x3, z2, z3 = m(g[0][1] ** 2), m(g[0][1] ** 3), m(g[2][2] ** 2), m(g[2][2] ** 3)
    return [m(u[0] ** 2 + u[1] ** 2 + u[2] ** 2), sij, x2, x3, z2, z3, x3 / x2**1.5, z3 / z2**1.5,
            float(u[0].numel())]


def exact(case, seed):
    cells = sum(nc**3 for nc in _sizes(case))
    if cells * (1 if case["kind"] in ("stats", "ensemble") else case["steps"]) > 8 * EXACT_CELLS:
        return None
    kind = case["kind"]
    if kind == "ensemble":
        out = [_step(W, case, _dt(W, case)) for W in _fields(case, seed)]
        return [torch.cat([W[q].reshape(-1) for W in out]) for q in range(5)]
    W = next(_fields(case, seed))
    if kind == "stats":
        return _stats(W, case)
    dt = _dt(W, case)
    lines = []
    if kind == "particles":
        x0, y0, z0 = torch.from_numpy(_positions(case, seed)).cuda()
        pos = [y0, x0, z0]
    for _ in range(case["steps"]):
        if kind == "loop":
            lines.append(_stats(W, case))
        if kind == "particles":
            values, grads = _props(W, pos)
            lines.append(_particle_line(values, grads))
            for a, b in enumerate((2, 1, 3)):  # y moves with v, x with u, z with w
                x = pos[a] + values[b] * dt
                x = torch.where(x > 2 * math.pi, x - 2 * math.pi, x)
                pos[a] = torch.where(x < 0, x + 2 * math.pi, x)
        W = _step(W, case, dt)
    if kind == "evolve":
        nt = [torch.arange(-3, n + 3, device="cuda") % n for n in W.shape[1:]]
        return W[:, nt[0]][:, :, nt[1]][:, :, :, nt[2]].cpu()
    arrays = [W[q] for q in range(5)]
    if kind == "loop":
        return {"lines": np.array(lines), "W": arrays}
    if kind == "particles":
        records = torch.stack(pos + values + [g for row in grads for g in row])
        return {"lines": np.array(lines), "records": records.cpu().numpy(), "W": arrays}
    return arrays
