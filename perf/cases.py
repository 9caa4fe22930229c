"""The work that is timed: one pass each through the framework's public entry points.

A case is a dict of plain values.  ``kind`` names the entry point:

- ``step``: ``RK3Integrator.step`` with its diagnostics read, as a driver's loop calls it.
- ``graph``: ``RK3Integrator.capture`` once, then one launch of the captured steps a pass, as
  the serving loop advances a resident run.  The state advances from pass to pass.
- ``projection``: ``AnelasticProjection.apply_projection`` (the pre-balance iterations).
- ``poisson``: ``VariableCoefficientPoissonSolver.solve``.
- ``advection`` / ``damping``: one slow component's ``compute_tendency``.
- ``readout``: ``compute_diagnostics`` of one state (the periodic log line).

``physics`` of the steps: ``lh82`` (WS5 advection, beta-plane, buoyancy, projection), ``heated``
(the same with eyewall heating) and ``production`` (``build_production_config``).  Inputs are a
Holland-type vortex with a warm core off the domain's centre, a background flow with eddies
and convective cells, and grid-scale noise, all from the seed.

``exact`` restates the algorithm in 64-bit torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

GRAVITY, R_D, C_P, P_REF = 9.81, 287.04, 1004.5, 100_000.0
F0, BETA = 4.99e-5, 2.15e-11
U_ENV, V_ENV = -3.0, 1.0
HEAT = dict(Q_max=3.0 / 3600.0, width_z=math.sqrt(2.0) * 2e3, z_peak=6e3)
# build_production_config's constants
NU4, EPSILON, TAU_COOL, CD, H_BL = 3.0e11, 0.5, 1800.0, 1.5e-3, 1000.0


def _case(kind, nx, ny, nz, precision, dx, dt=None, Lz=16e3, physics="lh82", nsteps=1):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=precision, dx=float(dx), Lz=float(Lz),
             physics=physics, nsteps=nsteps)
    c["dt"] = float(dt if dt is not None else dx / 100.0)
    return c


def listed():
    return [
        # the idealised beta-drift run, FP64 throughout (the default precision)
        dict(_case("step", 128, 128, 32, "fp64", 20e3, 60.0), name="drift_128_fp64"),
        # the mid-size heated run in both precisions that a study compares
        dict(_case("step", 512, 512, 64, "fp64", 5e3, 40.0, physics="heated"),
             name="heated_512_fp64"),
        dict(_case("step", 512, 512, 64, "fp32r", 5e3, 40.0, physics="heated"),
             name="heated_512_fp32r"),
        # the production-size single run of the benchmark, FP32 state with its defect correction
        dict(_case("step", 1024, 1024, 80, "fp32r", 4e3, 30.0, Lz=20e3), name="large_1024_fp32r"),
        # a storm replay with the production physics on one of the standard grids
        dict(_case("step", 320, 320, 32, "fp64", 15_625.0, 30.0, Lz=20e3, physics="production"),
             name="storm_320_fp64"),
        # one resident run of a served ensemble: captured steps, one launch a pass
        dict(_case("graph", 192, 192, 48, "fp32r", 10e3, 120.0, physics="production", nsteps=2),
             name="served_192_fp32r"),
        # the smallest ensemble member, where launches and latency count
        dict(_case("step", 96, 96, 32, "fp32", 10e3, 80.0), name="member_96_fp32"),
        # a pre-balance projection of a standard grid, FP64
        dict(_case("projection", 384, 384, 48, "fp64", 10e3), name="prebalance_384_fp64"),
        # the same on an odd level count and ragged, radix-3 and radix-5 lengths
        dict(_case("projection", 250, 162, 45, "fp32", 12e3), name="prebalance_ragged_fp32"),
        # a bare elliptic solve (initialisation, potential recovery)
        dict(_case("poisson", 256, 240, 40, "fp64", 8e3), name="poisson_256_fp64"),
        # the advection component alone (budget diagnostics)
        dict(_case("advection", 360, 300, 60, "fp32", 6e3), name="advection_360_fp32"),
        # the diagnostics log line of a mid-size state
        dict(_case("readout", 512, 512, 64, "fp32", 5e3), name="readout_512_fp32"),
    ]


def _smooth(lo, hi):
    """Even lengths in [lo, hi] whose half has no factor above 5."""
    out = []
    for n in range(lo, hi + 1, 2):
        m = n // 2
        for p in (2, 3, 5):
            while m % p == 0:
                m //= p
        if m == 1:
            out.append(n)
    return out


def draw(rng):
    kind = rng.choice(["step", "step", "step", "graph", "projection", "projection", "poisson",
                       "advection", "damping", "readout"])
    fp32 = "fp32r" if kind in ("step", "graph") else "fp32"
    precision = rng.choice(["fp64", fp32, "fp32"])
    physics = rng.choice(["lh82", "heated", "production"]) if kind in ("step", "graph") else "lh82"
    lengths = _smooth(64, 1024)

    def length():
        want = math.exp(rng.uniform(math.log(64), math.log(1024)))
        return min(lengths, key=lambda n: abs(math.log(n / want)))

    nx = length()
    ny = nx if rng.random() < 0.5 else length()
    nz = rng.randint(16, 96)
    most = 12_000_000 if precision == "fp64" else 40_000_000
    while nx * ny * nz > most:
        if nz > 48:
            nz = rng.randint(16, 48)
        elif nx >= ny:
            nx = max(n for n in lengths if n < nx)
        else:
            ny = max(n for n in lengths if n < ny)
    dx = rng.choice([4e3, 5e3, 8e3, 10e3] + ([15_625.0, 20e3] if precision == "fp64" else []))
    nsteps = 2 if kind == "graph" else 1
    return _case(kind, nx, ny, nz, precision, dx, Lz=rng.choice([16e3, 20e3]), physics=physics,
                 nsteps=nsteps)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _dtype(case):
    return torch.float64 if case["precision"] == "fp64" else torch.float32


def _column(case):
    """(z, rho0, theta0) of the standard base state, host FP64."""
    nz, dz = case["nz"], case["Lz"] / case["nz"]
    z = (np.arange(nz) + 0.5) * dz
    theta0 = 300.0 * np.exp(0.01 ** 2 * z / GRAVITY)
    exner = np.empty(nz)
    exner[0] = 1.0 - (GRAVITY / C_P) * z[0] / theta0[0]
    for k in range(nz - 1):
        exner[k + 1] = exner[k] - (GRAVITY / C_P) * (0.5 * dz) * (1.0 / theta0[k]
                                                                  + 1.0 / theta0[k + 1])
    return z, P_REF * exner ** (C_P / R_D) / (R_D * theta0 * exner), theta0


def _fields(case, seed):
    """u, v, w, theta' on the device in the case's type, from the seed alone."""
    nx, ny, nz, dx = case["nx"], case["ny"], case["nz"], case["dx"]
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(int(seed) * 7919 + 17)
    r = np.random.RandomState(int(seed) % (1 << 31))
    f = dict(dtype=torch.float64, device=dev)
    z = (torch.arange(nz, **f) + 0.5) * (case["Lz"] / nz)
    zh = torch.arange(nz + 1, **f) * (case["Lz"] / nz)
    rho = torch.as_tensor(_column(case)[1], **f)
    rho_h = torch.cat([rho[:1], 0.5 * (rho[:-1] + rho[1:]), rho[-1:]])

    def noise(levels, size):
        return (torch.rand((nx, ny, levels), generator=g, **f) * 2.0 - 1.0) * size

    # the vortex: Holland's profile, tapered to calm at the domain's edge
    vmax, b = r.uniform(40, 50), r.uniform(1.6, 2.0)
    rmax = max(50e3, 4 * dx) * r.uniform(1.0, 1.25)
    x = (torch.arange(nx, **f) + 0.5) * dx - nx * dx * r.uniform(0.4, 0.6)
    y = (torch.arange(ny, **f) + 0.5) * dx - ny * dx * r.uniform(0.4, 0.6)
    rad = torch.sqrt(x[:, None] ** 2 + y[None, :] ** 2).clamp_min(1.0)
    p = (rmax / rad) ** b
    edge = torch.clamp(rad / (0.45 * min(nx, ny) * dx), max=1.0)
    vt = vmax * torch.sqrt(p * torch.exp(1.0 - p)) * 0.5 * (1.0 + torch.cos(math.pi * edge))
    decay = torch.clamp(1.0 - z / 14e3, min=0.0)
    u = (-vt * y[None, :] / rad)[:, :, None] * decay + U_ENV + noise(nz, 0.02)
    v = (vt * x[:, None] / rad)[:, :, None] * decay + V_ENV + noise(nz, 0.02)
    w = torch.zeros((nx, ny, nz + 1), **f)
    th = 0.3 * torch.exp(-(rad / (1.5 * rmax)) ** 2)[:, :, None] * torch.sin(
        math.pi * z / case["Lz"]) + noise(nz, 0.02)
    # the environment: a few periodic modes, each an eddy (rotational, 8 m/s) and a convective
    # cell (low-level inflow under the updraught, its mass flux closed by w, which a projection
    # alone starts without)
    m = math.pi / case["Lz"]
    updraught = 0.6 if case["kind"] == "projection" else min(0.8, 0.3 + 0.4 * dx / 10e3)
    for _ in range(3):
        kx = 2.0 * math.pi * max(1, round(nx / r.uniform(8, 16))) / (nx * dx)
        ky = 2.0 * math.pi * max(1, round(ny / r.uniform(8, 16))) / (ny * dx)
        px, py = kx * x + r.uniform(0, 6), ky * y + r.uniform(0, 6)
        cx, sx, cy, sy = torch.cos(px), torch.sin(px), torch.cos(py), torch.sin(py)
        eddy = 8.0 / math.hypot(kx, ky) * decay
        cell = updraught * m / (kx * kx + ky * ky) * (torch.cos(m * z) / rho)
        up = (cx[:, None] * cy[None, :])[:, :, None]
        ss = (sx[:, None] * sy[None, :])[:, :, None]
        u += -kx * (sx[:, None] * cy[None, :])[:, :, None] * cell + ky * up * eddy
        v += -ky * (cx[:, None] * sy[None, :])[:, :, None] * cell + kx * ss * eddy
        if case["kind"] != "projection":
            w += updraught * up * (torch.sin(m * zh) / rho_h)
        th += 0.15 * up * torch.sin(m * z)
    w[:, :, 0] = 0.0
    w[:, :, -1] = 0.0
    return [a.to(_dtype(case)).contiguous() for a in (u, v, w, th)]


def _sizes(case):
    nx, ny, nz, dx = case["nx"], case["ny"], case["nz"], case["dx"]
    return nx, ny, nz, nx * dx, ny * dx, case["Lz"]


def _heating(case):
    return dict(HEAT, r_eyewall=max(40e3, 3 * case["dx"]),
                width_r=math.sqrt(2.0) * max(15e3, 2 * case["dx"]))


def _config(case):
    from oraclev8_b200.grid import LorenzStaggering
    from oraclev8_b200.production_config import build_production_config
    from oraclev8_b200.solver import (AdvectionComponent, AnelasticProjection, BuoyancyComponent,
                                      CoriolisComponent, DiabaticHeatingComponent,
                                      LH82AnelasticEquationSet, OperatorConfig)
    nx, ny, nz, Lx, Ly, Lz = _sizes(case)
    if case["physics"] == "production":
        return build_production_config(nx, ny, nz, Lx, Ly, Lz, F0, U_ENV, V_ENV)
    kw = dict(equation_set=LH82AnelasticEquationSet(), staggering=LorenzStaggering(),
              buoyancy=BuoyancyComponent(),
              projection=AnelasticProjection(nx, ny, nz, Lx, Ly, Lz),
              advection=AdvectionComponent(nx, ny, nz, Lx, Ly, Lz, scheme="upwind5h"),
              coriolis=CoriolisComponent(f=F0, mode="beta_plane", beta=BETA, Ly=Ly, ny=ny,
                                         u_env=U_ENV, v_env=V_ENV, periodic_taper=True))
    if case["physics"] == "heated":
        kw["diabatic_heating"] = DiabaticHeatingComponent(nx=nx, ny=ny, nz=nz, Lx=Lx, Ly=Ly,
                                                          Lz=Lz, **_heating(case))
    return OperatorConfig(**kw)


def prepare(case, seed):
    from oraclev8_b200.production_config import BaseState
    from oraclev8_b200.solver import (AdvectionComponent, AnelasticProjection,
                                      HelmholtzDivergenceDampingComponent, RK3Integrator, State,
                                      VariableCoefficientPoissonSolver)
    nx, ny, nz, Lx, Ly, Lz = _sizes(case)
    kind = case["kind"]
    base = BaseState(nz, Lz)
    s = dict(case=case, base=base)
    u, v, w, th = _fields(case, seed)
    s["state"] = State(u, v, w, th, torch.zeros_like(u), 0.0)
    if kind in ("step", "graph"):
        s["integrator"] = RK3Integrator(_config(case), base, precision=case["precision"])
        if kind == "graph":
            s["graph"] = s["integrator"].capture(s["state"], case["dt"], case["nsteps"])
    elif kind == "projection":
        s["component"] = AnelasticProjection(nx, ny, nz, Lx, Ly, Lz)
    elif kind == "advection":
        s["component"] = AdvectionComponent(nx, ny, nz, Lx, Ly, Lz, scheme="upwind5h")
    elif kind == "damping":
        s["component"] = HelmholtzDivergenceDampingComponent(EPSILON, Lx, Ly, nx, ny)
    elif kind == "poisson":
        s["solver"] = VariableCoefficientPoissonSolver(nx, ny, nz, Lx, Ly, Lz)
        s["rhs"] = _rhs(case, u, v, w)
        rh = np.concatenate([base.rho0[:1], 0.5 * (base.rho0[:-1] + base.rho0[1:]),
                             base.rho0[-1:]])
        s["rho"] = (base.rho0, rh)
    return s


def _rhs(case, u, v, w):
    """A source of the size and spectrum of the state's divergence, whose sum is zero."""
    d = ((torch.roll(u, -1, 0) - torch.roll(u, 1, 0)) / (2.0 * case["dx"])
         + (torch.roll(v, -1, 1) - torch.roll(v, 1, 1)) / (2.0 * case["dx"])
         + (w[:, :, 1:] - w[:, :, :-1]) * (case["nz"] / case["Lz"]))
    return d.contiguous()


def run(s):
    case, st = s["case"], s["state"]
    kind = case["kind"]
    if kind == "step":
        out, dg = s["integrator"].step(st, case["dt"])
        got = dict(u=out.u, v=out.v, w=out.w, theta=out.theta_prime,
                   phi=out.projection_potential, max_u=dg.max_u, max_v=dg.max_v,
                   max_w=dg.max_w, max_theta=dg.max_theta_prime)
        if case["precision"] == "fp64":
            # the potential's surface extremes about its mean are differences of close numbers,
            # which single precision leaves a few digits
            got.update(phi_min=dg.surface_phi_min, phi_max=dg.surface_phi_max)
        return got
    if kind == "graph":
        s["graph"].launch()
        return dict(u=st.u, v=st.v, w=st.w, theta=st.theta_prime, phi=st.projection_potential)
    if kind == "projection":
        from oraclev8_b200.solver import State
        out = s["component"].apply_projection(
            State(st.u, st.v, st.w, st.theta_prime, st.projection_potential, st.t), None, None,
            s["base"], case["dt"])
        return dict(u=out.u, v=out.v, w=out.w, phi=out.projection_potential)
    if kind == "poisson":
        return dict(phi=s["solver"].solve(s["rhs"], *s["rho"], log_diagnostics=False).phi)
    if kind == "readout":
        from oraclev8_b200.diagnostics import compute_diagnostics
        return compute_diagnostics(st, s["base"], 0.5 * case["nx"] * case["dx"],
                                   0.5 * case["ny"] * case["dx"], case["dx"], case["dx"],
                                   U_ENV, V_ENV)
    t = s["component"].compute_tendency(st, None, None, s["base"], case["dt"])
    if kind == "damping":
        return dict(du=t.du_dt, dv=t.dv_dt)
    return dict(du=t.du_dt, dv=t.dv_dt, dw=t.dw_dt, dtheta=t.dtheta_prime_dt)


def work(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n, size = nx * ny * nz, 8 if case["precision"] == "fp64" else 4
    wn = nx * ny * (nz + 1)
    # one projection: three real transforms along x and two complex ones along y, and back
    # (real transforms at half a complex one's operations), the solve's two sweeps, the update
    transform = 2.5 * math.log2(nx) * 3 * 2 + 2.5 * math.log2(ny) * 3
    projection = n * (transform + 10 + 20)
    slow = n * (150 if case["physics"] != "production" else 120)
    state = (3 * n + wn) * size
    kind = case["kind"]
    if kind in ("step", "graph"):
        nproj = 3 if case["physics"] == "production" else 5
        nproj += 1 if case["precision"] == "fp32r" else 0
        k = case["nsteps"]
        return dict(bytes=2 * state + n * size, flops=k * (nproj * projection + 2 * slow))
    if kind == "projection":
        return dict(bytes=(5 * n + 2 * wn) * size, flops=projection)
    if kind == "poisson":
        return dict(bytes=2 * n * size, flops=n * (5 * math.log2(nx * ny) + 10))
    if kind == "advection":
        return dict(bytes=2 * state, flops=n * 140)
    if kind == "damping":
        return dict(bytes=4 * n * size, flops=n * (10 * math.log2(nx * ny) + 8))
    return dict(bytes=2 * n * size, flops=n * 12)


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

class _Exact:
    """The algorithm on double fields, plain torch: (nx, ny, nz) arrays, periodic in x and y."""

    def __init__(self, case):
        self.case = case
        self.nx, self.ny, self.nz, self.Lx, self.Ly, self.Lz = _sizes(case)
        self.dx, self.dz = case["dx"], case["Lz"] / case["nz"]
        f = dict(dtype=torch.float64, device="cuda")
        z, rho, th = _column(case)
        self.z, self.rho, self.th0 = (torch.as_tensor(a, **f) for a in (z, rho, th))
        self.rho_h = torch.cat([self.rho[:1], 0.5 * (self.rho[:-1] + self.rho[1:]),
                                self.rho[-1:]])
        k = lambda n: 2.0 * math.pi * torch.fft.fftfreq(n, d=self.dx, **f)  # noqa: E731
        self.kx, self.ky = k(self.nx)[:, None, None], k(self.ny)[None, :, None]

    # -- horizontal spectra ---------------------------------------------------
    @staticmethod
    def fft(a):
        return torch.fft.fft2(a, dim=(0, 1))

    @staticmethod
    def ifft(a):
        return torch.fft.ifft2(a, dim=(0, 1)).real

    # -- elliptic solve -------------------------------------------------------
    def solve(self, d):
        dh = self.fft(d).permute(2, 0, 1).contiguous()
        dh[:, 0, 0] -= dh[:, 0, 0].sum() / self.nz
        lo, up = self.rho_h[:-1] / self.dz ** 2, self.rho_h[1:] / self.dz ** 2
        lo = torch.cat([torch.zeros_like(lo[:1]), lo[1:]])
        up = torch.cat([up[:-1], torch.zeros_like(up[:1])])
        k2 = (self.kx ** 2 + self.ky ** 2)[:, :, 0].clone()
        k2[0, 0] = 1.0
        mean = dh[:, 0, 0].clone()
        gains = []
        for k in range(self.nz):
            den = -(lo[k] + up[k]) - k2 * self.rho[k]
            if k:
                den = den - lo[k] * gains[-1]
                dh[k] = (dh[k] - lo[k] * dh[k - 1]) / den
            else:
                dh[k] = dh[k] / den
            gains.append(up[k] / den)
        for k in range(self.nz - 2, -1, -1):
            dh[k] = dh[k] - gains[k] * dh[k + 1]
        # the horizontal mean: phi = 0 at the lowest level, the others from their own rows
        a = (torch.diag(-(lo + up)) + torch.diag(up[:-1], 1) + torch.diag(lo[1:], -1)).cpu()
        low = torch.linalg.solve(a[1:, 1:].to(torch.complex128), mean.cpu()[1:])
        dh[0, 0, 0] = 0.0
        dh[1:, 0, 0] = low.to(dh.device)
        return self.ifft(dh.permute(1, 2, 0))

    def project(self, u, v, w):
        r = self.rho
        div = self.ifft(1j * self.kx * self.fft(r * u) + 1j * self.ky * self.fft(r * v))
        flux = self.rho_h * w
        phi = self.solve(div + (flux[:, :, 1:] - flux[:, :, :-1]) / self.dz)
        ph = self.fft(phi)
        u = u - self.ifft(1j * self.kx * ph)
        v = v - self.ifft(1j * self.ky * ph)
        w = w.clone()
        w[:, :, 1:-1] -= (phi[:, :, 1:] - phi[:, :, :-1]) / self.dz
        return u, v, w, phi

    # -- slow terms -----------------------------------------------------------
    def ddz(self, q):
        mid = (q[:, :, 2:] - q[:, :, :-2]) / (2.0 * self.dz)
        return torch.cat([(q[:, :, 1:2] - q[:, :, :1]) / self.dz, mid,
                          (q[:, :, -1:] - q[:, :, -2:-1]) / self.dz], dim=2)

    def upwind(self, q, a, axis):
        """Fifth-order upwind-biased derivative along the flow (non-negative: from below)."""
        at = lambda o: torch.roll(q, -o, axis)  # noqa: E731
        below = -2 * at(-3) + 15 * at(-2) - 60 * at(-1) + 20 * q + 30 * at(1) - 3 * at(2)
        above = 2 * at(3) - 15 * at(2) + 60 * at(1) - 20 * q - 30 * at(-1) + 3 * at(-2)
        return torch.where(a >= 0, below, above) / (60.0 * self.dx)

    def centred(self, q, a, axis):
        return (torch.roll(q, -1, axis) - torch.roll(q, 1, axis)) / (2.0 * self.dx)

    def advection(self, u, v, w, th, ddx):
        ends = lambda q: torch.cat([q[:, :, :1], 0.5 * (q[:, :, :-1] + q[:, :, 1:]),  # noqa: E731
                                    q[:, :, -1:]], dim=2)
        wc, uh, vh = 0.5 * (w[:, :, :-1] + w[:, :, 1:]), ends(u), ends(v)
        total = self.th0[None, None, :] + torch.zeros_like(th[:1, :1])

        def along(q):
            return -(u * ddx(q, u, 0) + v * ddx(q, v, 1) + wc * self.ddz(q))

        dw = -(uh * ddx(w, uh, 0) + vh * ddx(w, vh, 1) + w * self.ddz(w))
        dw[:, :, 0] = 0.0
        dw[:, :, -1] = 0.0
        return along(u), along(v), dw, along(th) - wc * self.ddz(total)

    def f_of_y(self):
        n, beta = self.ny, BETA
        if self.case["physics"] == "production":
            omega = 7.2921e-5
            beta = 2.0 * omega * math.cos(math.asin(F0 / (2.0 * omega))) / 6.371e6
        dev = beta * ((torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) * self.dx
                      - 0.5 * self.Ly)
        m = max(1, int(round(0.20 * n)))
        taper = torch.ones_like(dev)
        ramp = torch.sin(math.pi * (torch.arange(m, dtype=torch.float64, device="cuda") + 0.5)
                         / (2.0 * m)) ** 2
        taper[:m] = ramp
        taper[n - m:] = ramp.flip(0)
        return (F0 + dev * taper)[None, :, None]

    def damping(self, u, v, dt):
        k2 = self.kx ** 2 + self.ky ** 2
        k2[0, 0] = 1.0
        psi = -(1j * self.kx * self.fft(u) + 1j * self.ky * self.fft(v)) / k2
        return tuple(-(EPSILON / dt) * self.ifft(1j * k * psi) for k in (self.kx, self.ky))

    def laplacian(self, q):
        return sum((torch.roll(q, 1, a) - 2.0 * q + torch.roll(q, -1, a)) / self.dx ** 2
                   for a in (0, 1))

    def heating(self):
        h = _heating(self.case)
        f = dict(dtype=torch.float64, device="cuda")
        x = (torch.arange(self.nx, **f) + 0.5) * self.dx - 0.5 * self.Lx
        y = (torch.arange(self.ny, **f) + 0.5) * self.dx - 0.5 * self.Ly
        rad = torch.sqrt(x[:, None] ** 2 + y[None, :] ** 2)
        ring = h["Q_max"] * torch.exp(-((rad - h["r_eyewall"]) / h["width_r"]) ** 2)
        return ring[:, :, None] * torch.exp(-((self.z - h["z_peak"]) / h["width_z"]) ** 2)

    def slow(self, u, v, w, th, dt):
        production = self.case["physics"] == "production"
        du, dv, dw, dth = self.advection(u, v, w, th, self.centred if production else self.upwind)
        f, up, vp = self.f_of_y(), u - U_ENV, v - V_ENV
        du, dv = du + f * vp, dv - f * up
        if production:
            rate = (CD * torch.sqrt(up[:, :, :1] ** 2 + vp[:, :, :1] ** 2) / self.dz
                    * torch.clamp(1.0 - self.z / H_BL, min=0.0))
            du, dv = du - rate * up, dv - rate * vp
            du = du - NU4 * self.laplacian(self.laplacian(u))
            dv = dv - NU4 * self.laplacian(self.laplacian(v))
            dth = dth - th / TAU_COOL
            hu, hv = self.damping(u, v, dt)
            du, dv = du + hu, dv + hv
        elif self.case["physics"] == "heated":
            dth = dth + self.heating()
        u, v, w, phi = self.project(u + dt * du, v + dt * dv, w + dt * dw)
        return u, v, w, th + dt * dth, phi

    def step(self, u, v, w, th):
        dt = self.case["dt"]
        u, v, w, th, _ = self.slow(u, v, w, th, 0.5 * dt)
        if self.case["physics"] == "production":
            u, v, w, fast = self.project(u, v, w)
        else:
            # the buoyancy is that of theta', which the fast stages leave alone, so the last
            # stage starts from the slow state and not from the stages before it
            b = GRAVITY * th / self.th0
            w = w.clone()
            w[:, :, 1:-1] += dt * 0.5 * (b[:, :, :-1] + b[:, :, 1:])
            u, v, w, fast = self.project(u, v, w)
        u, v, w, th, phi = self.slow(u, v, w, th, 0.5 * dt)
        return u, v, w, th, phi, fast


def _readout(e, u, v):
    """The log line's values: vorticity centre, peak winds, ring-mean flow, energies."""
    dx, z = e.dx, e.z
    low = z <= 3000.0
    ub, vb = u[:, :, low].mean(2), v[:, :, low].mean(2)
    zeta = ((torch.roll(vb, -1, 0) - torch.roll(vb, 1, 0))
            - (torch.roll(ub, -1, 1) - torch.roll(ub, 1, 1))) / (2.0 * dx)
    x = (torch.arange(e.nx, dtype=torch.float64, device=u.device) + 0.5) * dx
    y = (torch.arange(e.ny, dtype=torch.float64, device=u.device) + 0.5) * dx

    def radius(cx, cy):
        return torch.sqrt((x[:, None] - cx) ** 2 + (y[None, :] - cy) ** 2)

    inside = radius(0.5 * e.nx * dx, 0.5 * e.ny * dx) < 200e3
    at = int(torch.argmax(torch.where(inside, zeta, torch.full_like(zeta, -math.inf))))
    cx, cy = float(x[at // e.ny]), float(y[at % e.ny])
    speed = torch.sqrt((u - U_ENV) ** 2 + (v - V_ENV) ** 2)
    below = torch.where(low, speed, torch.full_like(speed, -1.0))
    peak, top = int(torch.argmax(below)), int(torch.argmax(speed))
    ix, iy, iz = peak // (e.ny * e.nz), (peak // e.nz) % e.ny, peak % e.nz
    deep = z <= 12000.0
    ud, vd = u[:, :, deep].mean(2), v[:, :, deep].mean(2)
    rad = radius(cx, cy)
    rings = []
    edges = np.linspace(0.0, 120e3, 13)
    for b in range(12):
        m = (rad >= edges[b]) & (rad < edges[b + 1])
        if bool(m.any()):
            rings.append((float(ud[m].mean()), float(vd[m].mean())))
    uv, vv = (float(np.mean([r[i] for r in rings])) for i in (0, 1))
    return dict(xv_m=cx, yv_m=cy, vmax_lowlvl=float(below.max()),
                r_vmax_km=math.hypot(float(x[ix]) - cx, float(y[iy]) - cy) / 1e3,
                z_vmax_m=float(z[iz]), vmax_3d=float(speed.max()), z_vmax3d_m=float(z[top % e.nz]),
                u_vent=uv, v_vent=vv, u_gyre=uv - U_ENV, v_gyre=vv - V_ENV,
                pert_ke=float(0.5 * (speed ** 2).mean()), enstrophy=float(0.5 * (zeta ** 2).mean()))


def exact(case, seed):
    kind = case["kind"]
    e = _Exact(case)
    u, v, w, th = _fields(case, seed)
    if kind == "poisson":
        return dict(phi=e.solve(_rhs(case, u, v, w).double()))
    u, v, w, th = (a.double() for a in (u, v, w, th))
    if kind == "step":
        u, v, w, th, phi, fast = e.step(u, v, w, th)
        surface = fast[:, :, 0] - fast.mean()
        top = lambda a: float(a.abs().max())  # noqa: E731
        got = dict(u=u, v=v, w=w, theta=th, phi=phi, max_u=top(u), max_v=top(v), max_w=top(w),
                   max_theta=top(th))
        if case["precision"] == "fp64":
            got.update(phi_min=float(surface.min()), phi_max=float(surface.max()))
        return got
    if kind == "graph":
        for _ in range(case["nsteps"]):
            u, v, w, th, phi, _ = e.step(u, v, w, th)
        return dict(u=u, v=v, w=w, theta=th, phi=phi)
    if kind == "projection":
        return dict(zip(("u", "v", "w", "phi"), e.project(u, v, w)))
    if kind == "readout":
        return _readout(e, u, v)
    if kind == "damping":
        return dict(zip(("du", "dv"), e.damping(u, v, case["dt"])))
    return dict(zip(("du", "dv", "dw", "dtheta"), e.advection(u, v, w, th, e.upwind)))
