"""Performance cases: what programs that use this package have it do, through its public entry points.

Each case is one pass over a seeded synthetic state that lives where such a program keeps it (on the GPU;
in page-locked host memory for the host-resident step):

  redi    the Redi step on a device-resident state: ``redi_step``, or ``redi_calc_coeffs`` followed by
          ``redi_apply_flux`` as the reference's driver calls them (``calls`` = "two")
  host    ``redi_step_host``: the same step on a host-resident state
  batch   ``RediBatch.step``: uneven regional domains in one persistent launch
  ale     ``ale_remap_step`` on layers that have drifted from their targets
  meke    ``meke_step_ext``

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare`` / ``run`` make and run
one, ``work`` gives the bytes and operations of a pass that no implementation can avoid, and ``exact`` the
outputs of one pass as plain torch computes them in 64 bits.
"""

from __future__ import annotations

import math
import random

import torch

from more_benchmarks_dc_ocean_b200 import ale_remap as A
from more_benchmarks_dc_ocean_b200 import ocean_meke as M
from more_benchmarks_dc_ocean_b200 import ocean_redi as R

DEV = "cuda"
F64 = torch.float64


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest Redi call a model makes (a coarse or regional grid): launches and latency count
        dict(name="redi_small", kind="redi", nx=128, ny=96, nz=25, ntr=2, precision="fp64", eos=1, calls="step"),
        # the reference's benchmark size, its two routines called in turn as its driver does
        dict(name="redi_ref_two_calls", kind="redi", nx=473, ny=297, nz=30, ntr=2, precision="fp64", eos=1,
             calls="two"),
        # the production size, T and S
        dict(name="redi_production", kind="redi", nx=1440, ny=1080, nz=75, ntr=2, precision="fp64", eos=1,
             calls="step"),
        # a biogeochemistry run: T, S and 32 passive tracers in mixed precision
        dict(name="redi_mixed_34_tracers", kind="redi", nx=720, ny=576, nz=50, ntr=34, precision="mixed", eos=1,
             calls="step"),
        # odd sizes, the Wright equation of state, a few passive tracers (an odd number)
        dict(name="redi_wright_odd", kind="redi", nx=361, ny=275, nz=51, ntr=5, precision="fp64", eos=2,
             calls="two"),
        # a model whose state lives on the host and is stepped on the GPU
        dict(name="redi_host_state", kind="host", nx=480, ny=361, nz=50, ntr=2, precision="fp64", eos=1, bands=8),
        # an ensemble of uneven regional domains with T, S and 4 passive tracers each
        dict(name="batch_regional", kind="batch", domains=12, shapes=11, ntr=6, precision="fp64"),
        # the ALE remap at the reference's benchmark size
        dict(name="ale_ref", kind="ale", nx=479, ny=303, nz=30, passive=0, method=3, ke=False),
        # the ALE remap on the production grid
        dict(name="ale_production", kind="ale", nx=1444, ny=1084, nz=75, passive=0, method=3, ke=False),
        # odd sizes, passive tracers and the kinetic-energy rescale
        dict(name="ale_tracers_ke", kind="ale", nx=243, ny=187, nz=50, passive=3, method=3, ke=True),
        # MEKE at the reference's benchmark size
        dict(name="meke_ref", kind="meke", nx=479, ny=303, nz=30, terms=False),
        # MEKE on the production grid with its optional terms on
        dict(name="meke_production", kind="meke", nx=1444, ny=1084, nz=75, terms=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["redi", "redi", "redi", "redi", "host", "batch", "ale", "ale", "ale", "meke"])
    if kind in ("redi", "host"):
        while True:
            c = dict(kind=kind, nx=_log(rng, 64, 1440), ny=_log(rng, 48, 1080), nz=rng.randint(10, 90),
                     ntr=rng.choice([2, 2, 2, 2, 3, 4, 5, 6, 8, 12, 20, 34]) if kind == "redi" else 2,
                     precision=rng.choice(["fp64", "fp64", "mixed"]), eos=rng.choice([1, 1, 1, 2]))
            if c["nx"] * c["ny"] * c["nz"] * (c["ntr"] + 2) <= (2.0e8 if kind == "redi" else 4.0e7):
                break
        if kind == "redi":
            c["calls"] = rng.choice(["step", "step", "two"])
        else:
            c["bands"] = rng.randint(2, 12)
        return c
    if kind == "batch":
        return dict(kind=kind, domains=rng.randint(3, 16), shapes=rng.randint(0, 10**6), ntr=rng.randint(2, 6),
                    precision=rng.choice(["fp64", "mixed"]))
    while True:
        c = dict(kind=kind, nx=_log(rng, 64, 1444), ny=_log(rng, 48, 1084), nz=rng.randint(10, 100))
        if c["nx"] * c["ny"] * c["nz"] <= 6.0e7:
            break
    if kind == "ale":
        c.update(passive=rng.choice([0, 0, 1, 2, 4]), method=rng.choice([3, 3, 3, 2]), ke=rng.random() < 0.3)
    else:
        c.update(terms=rng.random() < 0.5)
    return c


# --------------------------------------------------------------------------------------------- Redi's inputs
_NGHOST, _DX, _DT, _KHTR = 2, 1.0e4, 1800.0, 1000.0


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFF)
    return g


def _depth(nxp, nyp, land, g):
    """Bathymetry of a 4000 m basin with seamounts whose common width gives the land fraction."""
    n = 40 if nxp * nyp > 200000 else 6
    nx, ny = nxp + 2 * _NGHOST, nyp + 2 * _NGHOST
    u = torch.rand(4, n, generator=g, device=DEV, dtype=F64)
    lx, ly = nxp * _DX, nyp * _DX
    cx, cy, amp = u[0] * lx, u[1] * ly, 4500.0 + 2000.0 * u[2]
    width = (0.5 + u[3]) * min(lx, ly)
    x = (torch.arange(nx, device=DEV, dtype=F64) - _NGHOST + 0.5) * _DX
    y = (torch.arange(ny, device=DEV, dtype=F64) - _NGHOST + 0.5) * _DX

    def at(xs, ys, s):
        sig = s * width[:, None]
        gx = torch.exp(-((xs[None] - cx[:, None]) ** 2) / (2.0 * sig * sig))
        gy = torch.exp(-((ys[None] - cy[:, None]) ** 2) / (2.0 * sig * sig))
        return 4000.0 - (amp[:, None] * gy).T @ gx

    step = max(1, min(nxp, nyp) // 128)
    xs, ys = x[_NGHOST:_NGHOST + nxp:step], y[_NGHOST:_NGHOST + nyp:step]
    lo, hi = 1e-4, 2.0
    for _ in range(24):
        s = 0.5 * (lo + hi)
        if float((at(xs, ys, s) < 50.0).double().mean()) < land:
            lo = s
        else:
            hi = s
    return at(x, y, 0.5 * (lo + hi)), x, y, lx, ly


def _box5(a):
    p = torch.nn.functional.pad(a[:, None], (2, 2, 2, 2), mode="replicate")
    return torch.nn.functional.avg_pool2d(p, 5, 1)[:, 0]


def _redi_problem(nxp, nyp, nz, ntr, eos, seed):
    """A seeded domain on the GPU: uneven layers over seamounts, stratified T and S with noise, smooth passive tracers."""
    g = _gen(seed)
    land = 0.30 if nxp * nyp > 200000 else 0.15
    depth, x, y, lx, ly = _depth(nxp, nyp, land, g)
    ny, nx = depth.shape
    wet = depth >= 50.0
    rnd = lambda: torch.randn(nz, ny, nx, generator=g, device=DEV, dtype=F64)  # noqa: E731
    h = (depth.clamp(min=0.0) / nz)[None] * (0.8 + 0.4 * torch.rand(nz, ny, nx, generator=g, device=DEV, dtype=F64))
    h.clamp_(min=1.0e-3)
    z = h.flip(0).cumsum(0).flip(0) - 0.5 * h
    horiz = 0.5 * torch.outer(torch.cos(2.0 * math.pi * y / ly), torch.sin(2.0 * math.pi * x / lx))
    tracers = [(2.0 + 23.0 * torch.exp(-z / 800.0) + horiz[None] + 0.05 * rnd()) * h,
               (34.5 + z / 4000.0 + 0.01 * rnd()) * h]
    for _ in range(ntr - 2):
        tracers.append(_box5(rnd()) * torch.exp(-z / 500.0) * h)
    wet_u = torch.zeros(ny, nx + 1, device=DEV, dtype=F64)
    wet_u[:, 1:nx] = (wet[:, :-1] & wet[:, 1:]).double()
    wet_v = torch.zeros(ny + 1, nx, device=DEV, dtype=F64)
    wet_v[1:ny] = (wet[:-1] & wet[1:]).double()
    full = lambda v, *s: torch.full(s, v, device=DEV, dtype=F64)  # noqa: E731
    return R.DeviceProblem(
        grid=R.HGrid(nx, ny, nxp, nyp, _NGHOST),
        metrics=R.OceanMetrics(full(_DX, ny, nx + 1), full(_DX, ny + 1, nx), full(1.0 / _DX, ny, nx + 1),
                               full(1.0 / _DX, ny + 1, nx), full(_DX * _DX, ny, nx), wet_u, wet_v),
        eos=R.OceanEos(1035.0, 10.0, 35.0, 2.0e-4, 7.6e-4, eos),
        ms=R.MultilayerState(nz, h, tracers, 1, 2),
        khtr_u_ext=full(_KHTR, ny, nx + 1), khtr_v_ext=full(_KHTR, ny + 1, nx), bc=R.OceanBC(), dt=_DT)


def _shapes(case):
    """(nx, ny, nz) of the regional domains: nx, ny log-uniform in [64, 512]."""
    rng = random.Random(case["shapes"])
    return [(_log(rng, 64, 512), _log(rng, 64, 512), rng.choice([25, 50, 75])) for _ in range(case["domains"])]


def _domains(case, seed):
    return [_redi_problem(a, b, c, case["ntr"], 1, seed * 1009 + k) for k, (a, b, c) in enumerate(_shapes(case))]


# ------------------------------------------------------------------------------------------ ALE's, MEKE's inputs
def _ale_problem(case, seed):
    """The reference benchmark's state (stretched sigma targets, bathymetry with vanished-layer columns, a free
    surface) with seeded phases, its layers drifted by up to 25 %."""
    g = _gen(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    ph = (2.0 * math.pi * torch.rand(6, generator=g, device=DEV, dtype=F64)).tolist()
    ar = lambda n: torch.arange(1, n + 1, device=DEV, dtype=F64)  # noqa: E731
    k = ar(nz)
    dsig = 1.0 + 3.0 * (k - 1.0) / max(1, nz - 1)
    dsig = dsig / dsig.sum()
    i, j = ar(nx)[None, :], ar(ny)[:, None]
    hbed = 15.0 + 4485.0 * (torch.sin(0.013 * i + ph[0]) * torch.cos(0.017 * j + ph[1])).abs()
    hbed = torch.where((i.long() + j.long()) % 97 == 0, torch.full_like(hbed, 3.0), hbed)
    eta = 0.4 * torch.sin(0.05 * i + 0.03 * j + ph[2])
    h = (hbed + eta)[None] * dsig[:, None, None] * (
        1.0 + 0.2 * torch.sin(3.0 * k[:, None, None] + (0.02 * i + 0.03 * j + ph[3])[None])
        + 0.05 * (2.0 * torch.rand(nz, ny, nx, generator=g, device=DEV, dtype=F64) - 1.0))
    h = h * ((hbed + eta) / h.sum(0))[None]
    kk = k[:, None, None]
    tr = [h * (2.0 + 12.0 * torch.exp(-(nz - kk) / 6.0) + 0.5 * torch.sin(0.02 * i)[None]), h * (34.5 + 0.8 * kk / nz)]
    for _ in range(case["passive"]):
        tr.append(h * torch.rand(nz, ny, nx, generator=g, device=DEV, dtype=F64))
    iu, jv = ar(nx + 1)[None, :], ar(ny + 1)[:, None]
    u = 0.3 * (torch.sin(0.01 * iu + ph[4]) * torch.cos(0.02 * j))[None] * (1.0 + 0.1 * kk)
    v = 0.2 * (torch.cos(0.015 * i + ph[5]) * torch.sin(0.018 * jv))[None] * (1.0 - 0.05 * kk)
    return dict(h=h, tracers=tr, u=u, v=v, eta=eta.contiguous(), hbed=hbed.contiguous(), dsig=dsig)


_MEKE_OUT = ("meke", "kh_diff", "le", "ku", "i_mass", "depth_tot", "bottom_fac2", "barotr_fac2", "src", "uflux",
             "vflux", "mass_ws")


def _meke_scalars(case):
    s = dict(gmcoeff=0.9, khcoeff=1.0, cdrag=2.5e-3, kh=100.0)
    if case["terms"]:
        s.update(cd_scale=0.3, min_gamma2=2.0e-2, uscale=0.02, alpha_rhines=0.15, alpha_frict=0.8, alpha_grid=0.4,
                 bgsrc=1.0e-9, frcoeff=0.5, damping=2.0e-6, khmeke_fac=0.7, backscatter=True, visc_coeff_ku=-0.25)
    return s


def _meke_problem(case, seed):
    g = _gen(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    uni = lambda lo, hi, *s: lo + (hi - lo) * torch.rand(*s, generator=g, device=DEV, dtype=F64)  # noqa: E731
    dx, dy = 8000.0 * uni(0.6, 1.4, ny, nx), 8000.0 * uni(0.6, 1.4, ny, nx)
    land = uni(0.0, 1.0, ny, nx) < 0.15
    h = uni(200.0, 5000.0, ny, nx)[None] / nz * uni(0.3, 1.7, nz, ny, nx)
    h = torch.where(land[None], uni(0.0, 1.0e-4, nz, ny, nx), h)
    y = torch.linspace(-1.0, 1.0, ny, device=DEV, dtype=F64)[:, None]
    d = dict(areaT=dx * dy, iareaT=1.0 / (dx * dy), idxT=1.0 / dx, idyT=1.0 / dy, dy_cu=8000.0 * uni(0.6, 1.4, ny, nx + 1),
             dx_cv=8000.0 * uni(0.6, 1.4, ny + 1, nx), idxCu=1.0 / (8000.0 * uni(0.6, 1.4, ny, nx + 1)),
             idyCv=1.0 / (8000.0 * uni(0.6, 1.4, ny + 1, nx)))
    s = dict(h_layer=h, rho_layer=uni(1020.0, 1030.0, nz, ny, nx), gm_src=uni(0.0, 2.0e-2, ny, nx),
             ke_diss_ext=-uni(0.0, 2.0e-3, ny, nx), meke=uni(0.0, 2.0e-2, ny, nx), kh_diff=uni(0.0, 300.0, ny, nx),
             f_centre=(1.0e-4 * y).abs().expand(ny, nx).contiguous(), u_bbl2=uni(0.0, 4.0e-2, ny, nx))
    return d, s


# --------------------------------------------------------------------------------------------- prepare and run
def _prec(case):
    return R.MIXED if case["precision"] == "mixed" else R.FP64


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("redi", "host"):
        dp = _redi_problem(case["nx"], case["ny"], case["nz"], case["ntr"], case["eos"], seed)
        s = dict(kind=kind, case=case, dp=dp, redi=R.make_redi(dp, _prec(case)))
        if kind == "host":
            pin = lambda t: torch.empty(t.shape, dtype=F64, pin_memory=True).copy_(t)  # noqa: E731
            s["host"] = R.MultilayerState(case["nz"], pin(dp.ms.h_layer), [pin(t) for t in dp.ms.tracers], 1, 2)
            dp.ms = None
        return s
    if kind == "batch":
        dps = _domains(case, seed)
        return dict(kind=kind, case=case, dps=dps, batch=R.RediBatch(dps, _prec(case)))
    if kind == "ale":
        p = _ale_problem(case, seed)
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        z3 = lambda: torch.zeros(nz, ny, nx, device=DEV, dtype=F64)  # noqa: E731
        z2 = lambda: torch.zeros(ny, nx, device=DEV, dtype=F64)  # noqa: E731
        vc = A.OceanVcoord(nz, p["dsig"], z3(), z3(), z2(), z2(), nx_total=nx, ny_total=ny, remap_method=case["method"],
                           remap_vel_conserve_ke=case["ke"])
        ms = A.AleState(nz, p["h"].clone(), p["tracers"], p["u"], p["v"], z3(), z3(), z3())
        return dict(kind=kind, case=case, grid=A.AleGrid(nx, ny), vc=vc, ms=ms, eta=p["eta"], hbed=p["hbed"],
                    drifted=p["h"])
    d, s = _meke_problem(case, seed)
    m = M.OceanMeke(**_meke_scalars(case), enable=True).init(case["nx"], case["ny"], case["nz"])
    for k in ("meke", "kh_diff", "f_centre", "u_bbl2"):
        m.arrays[k] = s[k]
    return dict(kind=kind, case=case, m=m, metrics=M.MekeMetrics(**d), gm=M.OceanGM(s["gm_src"]),
                ms=M.MekeLayers(case["nz"], s["h_layer"], s["rho_layer"]), ke=s["ke_diss_ext"])


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "redi":
        dp, redi = state["dp"], state["redi"]
        if case["calls"] == "step":
            R.redi_step(dp.grid, dp.metrics, dp.eos, redi, dp.ms, dp.dt, dp.khtr_u_ext, dp.khtr_v_ext, dp.bc)
        else:
            R.redi_calc_coeffs(dp.grid, dp.metrics, dp.eos, redi, dp.ms)
            R.redi_apply_flux(dp.grid, dp.metrics, redi, dp.ms, dp.dt, dp.khtr_u_ext, dp.khtr_v_ext, dp.bc)
        return dp.ms.tracers
    if kind == "host":
        dp, hs = state["dp"], state["host"]
        R.redi_step_host(dp.grid, dp.metrics, dp.eos, state["redi"], hs, dp.dt, dp.khtr_u_ext, dp.khtr_v_ext, dp.bc,
                         case["bands"])
        return hs.tracers
    if kind == "batch":
        state["batch"].step()
        dps = state["dps"]
        # one tensor per tracer over all domains would be a copy: whole fields of the domains, at most 64 outputs
        return [t for dp in dps for t in dp.ms.tracers][:64]
    if kind == "ale":
        ms, vc = state["ms"], state["vc"]
        ms.h_layer.copy_(state["drifted"])  # the dynamics between two remaps move the layers off their targets
        A.ale_remap_step(state["grid"], vc, ms, state["eta"], state["hbed"])
        return dict(h=ms.h_layer, tracers=ms.tracers, u=ms.u_face_x_layer, v=ms.v_face_y_layer,
                    mass=ms.mass_budget_remap, heat=ms.heat_budget_remap, salt=ms.salt_budget_remap, eta=state["eta"])
    m = state["m"]
    M.meke_step_ext(case["nx"], case["ny"], case["nz"], m, state["metrics"], state["gm"], state["ms"], 1800.0,
                    state["ke"])
    return {k: m.arrays[k] for k in _MEKE_OUT}


# --------------------------------------------------------------------------------------------------- the work
def _redi_work(nx, ny, nz, ntr, mixed):
    n2, ns = (nx + 2 * _NGHOST) * (ny + 2 * _NGHOST), 2 * nz + 2
    # thickness and tracers read, tracers written, both directions' coefficients written, the 2-D fields read
    b = 8.0 * n2 * nz * (1 + 2 * ntr) + 2.0 * n2 * ns * (24 if mixed else 32) + 8.0 * n2 * 13
    # per face surface: three density differences, a position, a thickness; per tracer a flux; per layer the edges
    return b, n2 * (2.0 * ns * (45 + 45 * ntr) + nz * 60.0 * ntr)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        ws = [_redi_work(a, b, c, case["ntr"], case["precision"] == "mixed") for a, b, c in _shapes(case)]
        return {"bytes": sum(w[0] for w in ws), "flops": sum(w[1] for w in ws)}
    if kind in ("redi", "host"):
        b, f = _redi_work(case["nx"], case["ny"], case["nz"], case["ntr"], case["precision"] == "mixed")
        return {"bytes": b, "flops": f}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n2, nu, nv = nx * ny, (nx + 1) * ny, nx * (ny + 1)
    if kind == "ale":
        ntr = 2 + case["passive"]
        # h read; h_old, target, h written; tracers, budgets and velocities read and written; 2-D fields
        return {"bytes": 8.0 * (nz * (n2 * (4 + 2 * ntr + 6) + 2 * nu + 2 * nv) + 5 * n2),
                "flops": nz * 80.0 * (n2 * ntr + nu + nv)}
    return {"bytes": 8.0 * (2 * nz * n2 + 24 * n2 + 4 * nu + 4 * nv), "flops": n2 * (3.0 * nz + 150.0)}


# -------------------------------------------------------------------------------- the outputs in plain torch
_G = 9.80665


def _edges(h, s):
    """Interface values of a column's scalar, top-down; h and s are (nk, ncol). PPM edges over limited slopes."""
    nk = h.shape[0]
    diff = torch.zeros_like(s)
    if nk > 2:
        a, b, c = h[:-2], h[1:-1], h[2:]
        inv = lambda x: torch.where(x != 0.0, 1.0 / x, x)  # noqa: E731
        sm, sc, sp = s[:-2], s[1:-1], s[2:]
        dc = (b * inv((a + c) + b)) * ((2.0 * a + b) * inv(c + b) * (sp - sc) + (2.0 * c + b) * inv(a + b) * (sc - sm))
        dl, dr = 2.0 * (sc - sm), 2.0 * (sp - sc)
        v = torch.copysign(torch.minimum(torch.minimum(dl.abs(), dc.abs()), dr.abs()), dc)
        diff[1:-1] = torch.where((torch.sign(dl) * torch.sign(dr) <= 0.0) | ~((c + b) * (a + b) > 0.0), 0.0, v)
    e = torch.empty(nk + 1, h.shape[1], device=h.device, dtype=F64)
    e[0] = s[0] - 0.5 * diff[0]
    e[nk] = s[nk - 1] + 0.5 * diff[nk - 1]
    if nk > 1:
        hk, hp = h[:-1], h[1:]
        hm = torch.cat([h[:1], h[:-2]])
        hq = torch.cat([h[2:], h[-1:]])
        ak, ap, pk, pp = s[:-1], s[1:], diff[:-1], diff[1:]
        r = 1.0 / (hk + hp)
        v = torch.where(hk < hp, ak + (hk * r) * (ap - ak), ap + (hp * r) * (ak - ap))
        r2, r3 = 1.0 / ((2.0 * hk + hp) + 1e-30), 1.0 / ((hk + 2.0 * hp) + 1e-30)
        f1 = 1.0 / ((hk + hp) + (hm + hq))
        f2 = 2.0 * (hp * hk) * r * ((hm + hk) * r2 - (hq + hp) * r3)
        f3, f4 = hk * (hm + hk) * r2, hp * (hp + hq) * r3
        v = v + f1 * (f2 * (ap - ak) - (f3 * pp - f4 * pk))
        e[1:nk] = torch.where(hk + hp <= 0.0, 0.5 * (ak + ap), v)
    return e


def _density(eos, T, S, p):
    """d(rho)/dT and d(rho)/dS of the linear or Wright (1997) equation of state."""
    if eos.variant == 1:
        rho = eos.rho0 + eos.beta_S * (S - eos.S_ref) - eos.alpha_T * (T - eos.T_ref)
        return -(rho * rho) * (eos.alpha_T / eos.rho0 ** 2), -(rho * rho) * (-eos.beta_S / eos.rho0 ** 2)
    a0, a1, a2 = 7.057924e-4, 3.480336e-7, -1.112733e-7
    b = (5.790749e8, 3.516535e6, -4.002714e4, 2.084372e2, 5.944068e5, -9.643486e3)
    c = (1.704853e5, 7.904722e2, -7.984422e0, 5.140652e-2, -2.302158e2, -3.079464e0)
    poly = lambda q: q[0] + q[1] * T + q[2] * T * T + q[3] * (T * T) * T + q[4] * S + q[5] * S * T  # noqa: E731
    p0, lam = poly(b), poly(c)
    P = p + p0
    rho = P / (lam + (a0 + a1 * T + a2 * S) * P)
    dT = lambda q: q[1] + 2.0 * q[2] * T + 3.0 * q[3] * T * T + q[5] * S  # noqa: E731
    dS = lambda q: q[4] + q[5] * T  # noqa: E731
    i = 1.0 / P
    return (-(rho * rho) * (a1 + dT(c) * i - lam * dT(b) * i * i), -(rho * rho) * (a2 + dS(c) * i - lam * dS(b) * i * i))


def _neutral(nk, cols, L, Rr, scale):
    """The neutral-surface sweep of faces between columns L and Rr: positions, layers and effective thicknesses."""
    T, S, dT, dS, P = cols
    ncol, ns = T.shape[1], 2 * nk + 2
    at = lambda X, k, c: X.view(-1)[(k - 1) * ncol + c]  # noqa: E731
    nf = L.numel()
    new = lambda v, dt=F64: torch.full((nf,), v, device=DEV, dtype=dt)  # noqa: E731
    kl, kr = new(1, torch.int64), new(1, torch.int64)
    lPl, lPr, lKl, lKr = new(0.0), new(0.0), kl.clone(), kr.clone()
    bottom, left = new(False, torch.bool), new(False, torch.bool)
    absL = absR = None
    out = []

    def drho(k1, c1, k2, c2):
        return 0.5 * ((at(dT, k1, c1) + at(dT, k2, c2)) * (at(T, k1, c1) - at(T, k2, c2)) +
                      (at(dS, k1, c1) + at(dS, k2, c2)) * (at(S, k1, c1) - at(S, k2, c2)))

    for s in range(ns):
        d = drho(kr, Rr, kl, L)
        pick = torch.where(d < 0.0, True, torch.where(d > 0.0, False, torch.where(kl + kr == 2, True, ~left)))
        left = torch.where(bottom, left, pick)
        sk, ak = torch.where(left, kl, kr), torch.where(left, kr, kl)
        sc, ac = torch.where(left, L, Rr), torch.where(left, Rr, L)
        km1 = (sk - 1).clamp(min=1)
        top, bot = drho(km1, sc, ak, ac), drho(km1 + 1, sc, ak, ac)
        pt, pb = at(P, km1, sc), at(P, km1 + 1, sc)
        gap = bot - top
        x = torch.where(gap > 0.0, (-top / gap).clamp(0.0, 1.0),
                        torch.where(top > 0.0, 0.0, torch.where(top < 0.0, 1.0, 0.5)))
        x = torch.where((pb > pt) & (gap >= 0.0), x, 0.5)
        x = torch.where(top >= bot, 1.0, x)
        x = torch.where(torch.where(left, top > 0.0, top >= 0.0) | (kl + kr == 2), 0.0, x)
        carry = (x >= 1.0) & (km1 < nk)
        ko, x = km1 + carry.long(), torch.where(carry, x - 1.0, x)
        lk, lp = torch.where(left, lKl, lKr), torch.where(left, lPl, lPr)
        back = (ko - lk).double() + (x - lp) < 0.0
        ko, x = torch.where(back, lk, ko), torch.where(back, lp, x)
        live = ak <= nk
        pa, ka = torch.where(live, 0.0, 1.0), torch.where(live, ak, nk)
        adv = live.long()
        kr, kl = torch.where(left, kr + adv, kr), torch.where(left, kl, kl + adv)
        bottom = bottom | ~live
        was = left
        left = torch.where(live, left, ~left)
        Pl, Pr = torch.where(was, x, pa), torch.where(was, pa, x)
        Kl, Kr = torch.where(was, ko, ka), torch.where(was, ka, ko)
        aL = at(P, Kl, L) + Pl * (at(P, Kl + 1, L) - at(P, Kl, L))
        aR = at(P, Kr, Rr) + Pr * (at(P, Kr + 1, Rr) - at(P, Kr, Rr))
        he = None
        if s:
            hL, hR = aL - absL, aR - absR
            he = torch.where(hL + hR > 0.0, 2.0 * hL * hR / (hL + hR), 0.0) * scale
        absL, absR, lPl, lPr, lKl, lKr = aL, aR, Pl, Pr, Kl, Kr
        out.append((Pl, Pr, Kl, Kr, he))
    return out


def _ppm_mean(xl, xr, aL, aR, m):
    dx, xa = xr - xl, 0.5 * (xr + xl)
    c = 2.0 * m - (aL + aR)
    return torch.where((dx > 0.0) & (dx <= 1.0), (aL + xa * ((aR - aL) + 3.0 * c)) - c * (xr * xr + xr * xl + xl * xl),
                       aL + (aR - aL) * xr + 3.0 * c * xr * (1.0 - xr))


def _redi_exact(dp):
    nx, ny, nk = dp.grid.nx_total, dp.grid.ny_total, dp.ms.nz_ml
    ncol = nx * ny
    top = lambda t: t.flip(0).reshape(nk, ncol)  # noqa: E731
    h = top(dp.ms.h_layer)
    he = h.clamp(min=1e-20)
    T, S = _edges(h, top(dp.ms.tracers[0]) / he), _edges(h, top(dp.ms.tracers[1]) / he)
    P = torch.zeros_like(T)
    for k in range(nk):
        P[k + 1] = P[k] + (_G * dp.eos.rho0) * h[k]
    dT, dS = _density(dp.eos, T, S, P)
    col = torch.arange(ncol, device=DEV).view(ny, nx)
    g0, e0, n0 = _NGHOST, _NGHOST + dp.grid.nx_phys, _NGHOST + dp.grid.ny_phys
    m, faces = dp.metrics, []
    for wet, L, Rr, wall, coef in (
            (m.wet_u[:, 1:nx], col[:, :-1], col[:, 1:], None,
             dp.dt * dp.khtr_u_ext[:, 1:nx] * m.dy_cu[:, 1:nx] * m.idxCu[:, 1:nx]),
            (m.wet_v[1:ny], col[:-1], col[1:], 0, dp.dt * dp.khtr_v_ext[1:ny] * m.dx_cv[1:ny] * m.idyCv[1:ny])):
        ok = wet > 0.0
        if wall is None:  # no flux through the walls of the physical domain
            ok[:, g0 - 1] = False
            ok[:, e0 - 1] = False
        else:
            ok[g0 - 1] = False
            ok[n0 - 1] = False
        at = ok.reshape(-1).nonzero()[:, 0]
        L, Rr, coef = L.reshape(-1)[at], Rr.reshape(-1)[at], coef.reshape(-1)[at]
        faces.append((L, Rr, coef, _neutral(nk, (T, S, dT, dS, P), L, Rr, 1.0 / (_G * dp.eos.rho0))))
    del T, S, dT, dS, P
    outs = []
    for tr in dp.ms.tracers:
        lay = top(tr) / he
        e = _edges(h, lay)
        aL, aR = e[:-1], e[1:]
        d = torch.copysign(torch.full_like(lay, 3.0), aR - aL) * ((lay - aL) + (lay - aR))
        flat = torch.sign(aR - lay) * torch.sign(lay - aL) <= 0.0
        big, small = d > (aR - aL).abs(), d < -(aR - aL).abs()
        aL, aR = (torch.where(flat, lay, torch.where(big, lay + 2.0 * (lay - aR), aL)),
                  torch.where(flat, lay, torch.where(small & ~big, lay + 2.0 * (lay - aL), aR)))
        tend = torch.zeros(nk * ncol, device=DEV, dtype=F64)
        at = lambda X, k, c: X.reshape(-1)[(k - 1) * ncol + c]  # noqa: E731
        for L, Rr, coef, sweep in faces:
            prev = None
            for Pl, Pr, Kl, Kr, eff in sweep:
                tl = (1.0 - Pl) * at(e, Kl, L) + Pl * at(e, Kl + 1, L)
                trr = (1.0 - Pr) * at(e, Kr, Rr) + Pr * at(e, Kr + 1, Rr)
                dbot = trr - tl
                if prev is not None:
                    Ql, Qr, Jl, Jr, dtop = prev
                    ml = _ppm_mean(Ql, Pl + (Kl - Jl).double(), at(aL, Jl, L), at(aR, Jl, L), at(lay, Jl, L))
                    mr = _ppm_mean(Qr, Pr + (Kr - Jr).double(), at(aL, Jr, Rr), at(aR, Jr, Rr), at(lay, Jr, Rr))
                    dl = mr - ml
                    no = (torch.sign(dtop) * torch.sign(dbot) <= 0.0) | (
                        torch.sign(0.5 * (dtop + dbot)) * torch.sign(dl) <= 0.0)
                    f = torch.where(no, 0.0, dl) * eff * coef
                    tend.index_add_(0, (Jl - 1) * ncol + L, f)
                    tend.index_add_(0, (Jr - 1) * ncol + Rr, -f)
                prev = (Pl, Pr, Kl, Kr, dbot)
        outs.append(tr + tend.view(nk, ny, nx).flip(0) * (1.0 / m.areaT)[None])
    return outs


def _remap(ho, hn, q, method):
    """Conservative remap of the layer means q from thicknesses ho to hn, all (nz, n): differences of the integral
    from the first interface."""
    nz, n = ho.shape
    if nz == 1:
        return q.clone()
    zo = torch.cat([torch.zeros_like(ho[:1]), ho.cumsum(0)])
    zn = torch.cat([torch.zeros_like(hn[:1]), hn.cumsum(0)])
    if method == 3 and nz > 2:
        e = 0.5 * (q[:-1] + q[1:])
        e[1:-1] = (7.0 / 12.0) * (q[1:-2] + q[2:-1]) - (1.0 / 12.0) * (q[:-3] + q[3:])
        l, r = torch.cat([q[:1], e]), torch.cat([e, q[-1:]])
        up, dn = torch.cat([q[:1], q[:-1]]), torch.cat([q[1:], q[-1:]])
        lo, hi = torch.minimum(torch.minimum(q, up), dn), torch.maximum(torch.maximum(q, up), dn)
        l, r = torch.maximum(lo, torch.minimum(hi, l)), torch.maximum(lo, torch.minimum(hi, r))
        dq, s6 = r - l, 6.0 * q - 3.0 * (l + r)
        flat, over = (q - l) * (r - q) <= 0.0, s6.abs() > dq.abs()
        l, r = (torch.where(flat, q, torch.where(over & (s6 * dq > 0.0), 3.0 * q - 2.0 * r, l)),
                torch.where(flat, q, torch.where(over & ~(s6 * dq > 0.0), 3.0 * q - 2.0 * l, r)))
        c6 = 6.0 * q - 3.0 * (l + r)
        part = lambda x, k: x * l.gather(0, k) + 0.5 * x * x * (r - l + c6).gather(0, k) - x ** 3 * c6.gather(0, k) / 3.0  # noqa: E731
    else:
        sl = torch.zeros_like(q)
        dl, dr = q[1:-1] - q[:-2], q[2:] - q[1:-1]
        sl[1:-1] = torch.where(dl * dr > 0.0, 0.5 * torch.copysign(torch.minimum(dl.abs(), dr.abs()), dl), 0.0)
        part = lambda x, k: x * q.gather(0, k) + (x * x - x) * sl.gather(0, k)  # noqa: E731
    cum = torch.cat([torch.zeros_like(q[:1]), (q * ho).cumsum(0)])
    k = torch.searchsorted(zo[1:].T.contiguous(), zn.T.contiguous(), right=True).T.clamp(max=nz - 1)
    d = ho.gather(0, k)
    x = torch.where(d > 0.0, (zn - zo.gather(0, k)) / d, 0.0).clamp(0.0, 1.0)
    F = cum.gather(0, k) + d * part(x, k)
    return torch.where(hn > 0.0, (F[1:] - F[:-1]) / hn, 0.0)


def _rescale(ho, hn, qo, qn):
    so, sn = ho.sum(0), hn.sum(0)
    bo, bn = (ho * qo).sum(0) / so, (hn * qn).sum(0) / sn
    ko, kn = (0.5 * ho * (qo - bo) ** 2).sum(0), (0.5 * hn * (qn - bn) ** 2).sum(0)
    f = torch.sqrt(ko / kn).clamp(0.0, 1.25)
    ok = (so > 1.5e-4) & (sn > 1.5e-4) & (ko > 0.0) & (kn > 0.0)
    return torch.where(ok[None], bn + f * (qn - bn), qn)


def _ale_exact(case, p):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    flat = lambda t: t.reshape(nz, -1)  # noqa: E731
    ho = flat(p["h"])
    hn = ho.sum(0)[None] * p["dsig"][:, None]
    tr = []
    for t in p["tracers"]:
        q = torch.where(ho > 1.5e-4, flat(t) / ho, 0.0)
        tr.append((_remap(ho, hn, q, case["method"]) * hn).view(nz, ny, nx))
    vel = []
    for q, ax in ((p["u"], 2), (p["v"], 1)):
        face = []
        for t in (ho.view(nz, ny, nx), hn.view(nz, ny, nx)):
            n = t.shape[ax]
            face.append(torch.cat([t.narrow(ax, 0, 1), 0.5 * (t.narrow(ax, 0, n - 1) + t.narrow(ax, 1, n - 1)),
                                   t.narrow(ax, n - 1, 1)], ax).reshape(nz, -1))
        r = _remap(face[0], face[1], flat(q), case["method"])
        vel.append((_rescale(face[0], face[1], flat(q), r) if case["ke"] else r).view(q.shape))
    h = hn.view(nz, ny, nx)
    return dict(h=h, tracers=tr, u=vel[0], v=vel[1], mass=h - p["h"], heat=tr[0] - p["tracers"][0],
                salt=tr[1] - p["tracers"][1], eta=hn.sum(0).view(ny, nx) - p["hbed"])


def _meke_exact(case, d, s):
    m = M.OceanMeke(**_meke_scalars(case))
    sdt = 1800.0 * m.dtscale
    h, rho, E = s["h_layer"], s["rho_layer"], s["meke"]
    mass, depth = (rho * h.clamp(min=1.5e-4)).sum(0), h.sum(0)
    im = torch.where(mass > 0.0, 1.0 / mass, 0.0)
    lfrict = depth / m.cdrag
    bf2 = (m.cd_scale ** 2 + (lfrict * m.cb > 0.0).double()).clamp(min=m.min_gamma2)
    tf2 = torch.ones_like(bf2)
    lgrid = torch.sqrt(d["areaT"])
    ueddy = torch.sqrt(2.0 * (tf2 * E).clamp(min=0.0))
    b = torch.zeros_like(E)
    f = s["f_centre"]
    b[:, 1:-1] += (0.5 * (f[:, 2:] - f[:, :-2]) * d["idxT"][:, 1:-1]) ** 2
    b[1:-1] += (0.5 * (f[2:] - f[:-2]) * d["idyT"][1:-1]) ** 2
    b = torch.sqrt(b)
    lrh = torch.where(b > 0.0, torch.sqrt(ueddy / b), 0.0)
    il = torch.zeros_like(E)
    for a, l in ((m.alpha_frict, lfrict), (m.alpha_rhines, lrh), (m.alpha_grid, lgrid)):
        il = il + torch.where(a * l > 0.0, 1.0 / (a * l), 0.0)
    le = torch.where(il > 0.0, 1.0 / il, 0.0)
    src = torch.full_like(E, m.bgsrc) + m.gmcoeff * im * s["gm_src"]
    if m.frcoeff >= 0.0:
        src = src - m.frcoeff * im * s["ke_diss_ext"]
    E = E + sdt * src

    def drag(E):
        rate = im * torch.sqrt(m.cdrag ** 2 * ((2.0 * bf2 * E).clamp(min=0.0) + s["u_bbl2"] + m.uscale ** 2))
        return E / (1.0 + 0.5 * sdt * torch.where(E < 0.0, 0.0, m.damping + rate * bf2))

    E = drag(E)

    def flux(ax, geo):
        n = E.shape[ax]
        lo, hi = (lambda t: t.narrow(ax, 0, n - 1)), (lambda t: t.narrow(ax, 1, n - 1))
        geo = geo.narrow(ax, 1, n - 1)
        k = m.kh + m.khmeke_fac * 0.5 * (lo(s["kh_diff"]) + hi(s["kh_diff"]))
        cap = 2.0 * sdt * (geo * torch.maximum(lo(d["iareaT"]), hi(d["iareaT"])))
        k = torch.where(k * cap > 0.25, 0.25 / cap, k)
        hm = 2.0 * lo(mass) * hi(mass) / ((lo(mass) + hi(mass)) + 1e-30)
        z = torch.zeros_like(E.narrow(ax, 0, 1))
        return torch.cat([z, (k * geo) * hm * (lo(E) - hi(E)), z], ax)

    uf, vf = flux(1, d["dy_cu"] * d["idxCu"]), flux(0, d["dx_cv"] * d["idyCv"])
    E = E + sdt * (d["iareaT"] * im) * ((uf[:, :-1] - uf[:, 1:]) + (vf[:-1] - vf[1:]))
    E = drag(E)
    kh = m.khcoeff * torch.sqrt(2.0 * (tf2 * E).clamp(min=0.0)) * le
    ku = m.visc_coeff_ku * torch.sqrt(2.0 * E.clamp(min=0.0)) * le if m.backscatter else torch.zeros_like(E)
    return dict(meke=E, kh_diff=kh, le=le, ku=ku, i_mass=im, depth_tot=depth, bottom_fac2=bf2, barotr_fac2=tf2,
                src=src, uflux=uf, vflux=vf, mass_ws=mass)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("redi", "host"):
        return _redi_exact(_redi_problem(case["nx"], case["ny"], case["nz"], case["ntr"], case["eos"], seed))
    if kind == "batch":
        return [t for dp in _domains(case, seed) for t in _redi_exact(dp)][:64]
    if kind == "ale":
        return _ale_exact(case, _ale_problem(case, seed))
    return _meke_exact(case, *_meke_problem(case, seed))
