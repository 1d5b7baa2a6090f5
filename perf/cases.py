"""The work whose speed is watched: what a user of this package has it do.

Two kinds of case.  Single operators, as a host model calls them
(``operators.Advection``, ``operators.VerticalDiffusion``, the internal
pressure of ``_pygetm``, ``simulation.TracerTransport``), and whole 3D steps
of a simulation replayed by ``ensemble.DomainRunner``.  Sizes run from a
small ensemble member to the 400 x 300 x 40 benchmark domain; the data types
are the three forms the entry points take: "fp64" (everything double),
"mixed" (float velocities and diffusivities, tracers stored in double) and
"f32" (float fields).
"""

from __future__ import annotations

import math

import numpy as np
import torch

from getm_gb300 import _pygetm, autotune, workloads
from getm_gb300.core import CENTERS, INTERFACES, Array, make_grids
from getm_gb300.domain import calculate_sigma, create_cartesian
from getm_gb300.ensemble import DomainRunner, make_member
from getm_gb300.operators import Advection, AdvectionScheme, AdvectionSplit, VerticalDiffusion
from getm_gb300.simulation import Fluxes, Simulation, TracerTransport
from getm_gb300.vertical_mixing import GOTM

F64 = torch.float64
DEV = "cuda"


def listed():
    return [
        # the smallest call: 2D advection of a depth-averaged field (a column
        # height or a 2D momentum component), launch-bound
        dict(name="adv2d_small", kind="adv2d", nx=97, ny=75, scheme=5, split=2),
        # biogeochemistry on an odd-sized coastal grid: several tracers in one
        # call, with horizontal diffusion and another limiter
        dict(name="adv3d_fp64_odd", kind="adv3d", nx=173, ny=131, nz=23, nt=6, scheme=1, diffusion=True, form="fp64"),
        # temperature and salinity of the benchmark domain, mixed form
        dict(name="adv3d_mixed", kind="adv3d", nx=400, ny=300, nz=40, nt=2, scheme=5, diffusion=False, form="mixed"),
        # implicit vertical viscosity/diffusivity with sources, double
        dict(name="vdiff_fp64", kind="vdiff", nx=200, ny=150, nz=30, nt=2, sources=True, cnpar=1.0, form="fp64"),
        # the tracers' vertical diffusion of the benchmark domain, mixed form
        dict(name="vdiff_mixed", kind="vdiff", nx=400, ny=300, nz=40, nt=2, sources=False, cnpar=1.0, form="mixed"),
        # internal pressure gradient, double (odd rows) and mixed form
        dict(name="ip_fp64", kind="ip", nx=251, ny=187, nz=33, form="fp64"),
        dict(name="ip_mixed", kind="ip", nx=400, ny=300, nz=40, form="mixed"),
        # the tracer-transport configuration: advection then diffusion of one
        # tracer through a prescribed flow, double
        dict(name="transport", kind="transport", nx=120, ny=100, nz=30),
        # one 3D step of an ensemble or serving member, mixed form
        dict(name="step_member", kind="step", setup="member", nx=92, ny=92, nz=20, split=24, nt=2, form="mixed"),
        # one 3D step of a tidally forced shelf sea with open boundaries
        dict(name="step_shelf", kind="step", setup="shelf", nx=240, ny=200, nz=20, split=6, nt=8, form="mixed"),
        # one 3D step of a wind-driven coastal domain with the turbulence
        # closure, double: the default form
        dict(name="step_coastal_fp64", kind="step", setup="coastal", nx=200, ny=150, nz=30, split=20, nt=2, form="fp64"),
        # one 3D step of the benchmark domain, mixed form
        dict(name="step_seamount", kind="step", setup="seamount", nx=400, ny=300, nz=40, split=30, nt=2, form="mixed"),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _within(most, nx, ny, nz, nt):
    """nx and nt such that nx ny nz (nt + 1) is at most ``most``."""
    nt = max(1, min(nt, most // (nx * ny * nz) - 1))
    return min(nx, most // (ny * nz * (nt + 1))), nt


def draw(rng):
    kind = rng.choice(["adv2d", "adv3d", "adv3d", "vdiff", "vdiff", "ip", "transport", "step"])
    nx, ny, nz = _spread(rng, 64, 400), _spread(rng, 64, 300), _spread(rng, 8, 40)
    if kind == "adv2d":
        return dict(kind=kind, nx=nx, ny=ny, scheme=rng.randint(1, 6), split=rng.randint(1, 3))
    if kind == "adv3d":
        nt, form = _spread(rng, 1, 8), rng.choice(["fp64", "mixed", "f32"])
        nx, nt = _within(3_600_000 if form == "fp64" else 14_400_000, nx, ny, nz, nt)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, nt=nt, scheme=rng.randint(1, 6), diffusion=rng.random() < 0.3,
                    form=form)
    if kind == "vdiff":
        nx, nt = _within(9_600_000, nx, ny, nz, _spread(rng, 1, 6))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, nt=nt, sources=rng.random() < 0.5,
                    cnpar=rng.choice([1.0, 1.0, 0.7]), form=rng.choice(["fp64", "mixed", "f32"]))
    if kind == "ip":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, form=rng.choice(["fp64", "mixed"]))
    if kind == "transport":
        return dict(kind=kind, nx=min(nx, 240), ny=min(ny, 200), nz=nz)
    setup = rng.choice(["member", "shelf", "coastal", "seamount"])
    case = dict(kind=kind, setup=setup, nx=nx, ny=ny, nz=nz, split=_spread(rng, 10, 30), nt=2, form="mixed")
    if setup == "member":
        case["nx"] = case["ny"] = min(nx, 256)
    elif setup == "shelf":
        case.update(nx=min(nx, 240), ny=min(ny, 200), split=6, nt=_spread(rng, 2, 12))
    elif setup == "coastal":
        case.update(nx=_within(1_800_000, min(nx, 220), min(ny, 160), nz, 1)[0], ny=min(ny, 160), form="fp64")
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _modes(rng, ny, nx, n=6, top=5):
    """Sum of n random Fourier modes of up to ``top`` waves, in [-1, 1] (numpy)."""
    y, x = np.arange(ny)[:, None] / ny, np.arange(nx)[None, :] / nx
    f = np.zeros((ny, nx))
    for _ in range(n):
        kx, ky = rng.integers(-top, top + 1, 2)
        f += rng.uniform(0.5, 1.0) * np.cos(2 * np.pi * (kx * x + ky * y) + rng.uniform(0, 2 * np.pi))
    return f / max(np.abs(f).max(), 1e-12)


def _host_grid(rng, nx, ny, nz, dx=1000.0):
    """A coastal domain: 10-100 m deep, about 15 % of it land."""
    H = 55.0 + 45.0 * _modes(rng, ny, nx)
    q = _modes(rng, ny, nx, top=8)
    mask = (q >= np.quantile(q, 0.15)).astype(int)
    x, y = dx * (np.arange(nx) + 0.5), dx * (np.arange(ny) + 0.5)
    dom = create_cartesian(x, y, mask=mask, H=H, f=1e-4, z0=0.01)
    return dom.create_grids(nz, halox=2, haloy=2, velocity_grids=2)


def _up(a, dtype=F64):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV, dtype)


def _grid(rng, nx, ny, nz, zoom=0.0):
    """Device grids with sigma layers (thicker in mid-water with zoom > 0).
    Land holds zeros rather than the huge fill value, here and in every field
    that comes back, so that a comparison of whole fields is one of water."""
    autotune.apply(None)  # the library's own launch shapes
    T = make_grids(_host_grid(rng, nx, ny, max(nz, 1)), DEV)
    dga = _up(calculate_sigma(max(nz, 1), zoom, zoom))[:, None, None]
    for g in T.all_grids():
        g.D.all_values.copy_(torch.where(g.mask.all_values != 0, g.D.all_values, 0.0))
        g.hn.all_values.copy_(dga * g.D.all_values)
        g.ho = Array(g, g.hn.all_values.clone(), z=CENTERS)
    h = T.hn.all_values
    zf = torch.cat([torch.zeros_like(h[:1]), h.cumsum(0)]) - T.D.all_values
    T.zf.all_values.copy_(zf)
    T.zc.all_values.copy_(0.5 * (zf[1:] + zf[:-1]))
    return T


def _wet(g):
    return (g.mask.all_values == 1) | (g.mask.all_values == 2)


def _flow(T, rng, nz):
    """Sheared horizontal velocities, zero on closed faces, and the vertical
    velocity relative to the sigma layers that continuity gives."""
    s = (torch.arange(nz, device=DEV, dtype=F64) + 0.5)[:, None, None] / max(nz, 1)
    shape = T.mask.all_values.shape
    out = []
    for g in (T.ugrid, T.vgrid):
        a, b = _up(_modes(rng, *shape)), _up(_modes(rng, *shape, top=12))
        v = 0.5 * a * (0.5 + s) + 0.15 * b * torch.cos(math.pi * s)
        out.append(torch.where(_wet(g), v, torch.zeros_like(v)))
    u, v = out
    pu = u * torch.where(_wet(T.ugrid), T.ugrid.hn.all_values, 0.0) * T.ugrid.dy.all_values
    pv = v * torch.where(_wet(T.vgrid), T.vgrid.hn.all_values, 0.0) * T.vgrid.dx.all_values
    pu, pv = torch.where(_wet(T.ugrid), pu, 0.0), torch.where(_wet(T.vgrid), pv, 0.0)
    div = torch.zeros_like(u)
    div[:, 1:, 1:] = pu[:, 1:, 1:] - pu[:, 1:, :-1] + pv[:, 1:, 1:] - pv[:, :-1, 1:]
    div = torch.where(T.mask.all_values == 1, div * T.iarea.all_values, 0.0)
    w = torch.zeros((nz + 1,) + tuple(shape), dtype=F64, device=DEV)
    w[1:] = -div.cumsum(0) + div.sum(0) * torch.arange(1, nz + 1, device=DEV, dtype=F64)[:, None, None] / nz
    w[nz] = 0.0
    return u, v, w


def _tracer(T, rng, nz, dtype):
    """A stratified field with a front and small-scale variability."""
    shape = T.mask.all_values.shape
    s = (torch.arange(nz, device=DEV, dtype=F64) + 0.5)[:, None, None] / nz
    front = torch.tanh(8.0 * _up(_modes(rng, *shape)) + 2.0 * (s - 0.5))
    f = 12.0 + 4.0 * s + 3.0 * front + 0.2 * _up(_modes(rng, *shape, top=40)) * torch.cos(9.0 * s)
    return torch.where(T.mask.all_values != 0, f, 0.0).to(dtype)


def _step_sim(case, seed):
    rng = np.random.default_rng(seed)
    if case["setup"] == "shelf":
        autotune.apply(None)
        # weak tides, a tidal viscosity and a short time step: the flow stays
        # within that step over thousands of passes
        wl = workloads.shelf_sea(nx=case["nx"], ny=case["ny"], nz=case["nz"], ntracer=case["nt"], seed=seed, umax=0.3,
                                 tide=0.25)
        wl.params.update(split_factor=case["split"], timestep=4.0, num=1e-2, nuh=1e-2)
        return workloads.start_shelf_sea(wl, case["form"], device=DEV)
    if case["setup"] == "member":
        n = case["nx"]
        wl = workloads.ensemble_member(rng, nmin=n, nmax=n, nzmin=case["nz"], nzmax=case["nz"])
        # a steady breeze: the members' strongest winds outrun their prescribed
        # viscosity within days, and these steps go on for weeks
        wl.params.update(split_factor=case["split"], taux=0.02)
        return make_member(wl, case["form"], device=DEV, tiles="auto")
    if case["setup"] == "seamount":
        wl = workloads.seamount(case["nx"], case["ny"], case["nz"], split_factor=case["split"])
        Th, dga, p, dt = wl.T, wl.dga, wl.params, wl.params["timestep"]
        sim = Simulation(Th, dga, num=p["num"], nuh=p["nuh"], precision=case["form"], airsea=Fluxes(), tiles="auto",
                         device=DEV)
        depth = 4500.0
    else:
        Th = _host_grid(rng, case["nx"], case["ny"], case["nz"])
        sim = Simulation(Th, calculate_sigma(case["nz"], 1.0, 1.0), precision=case["form"], airsea=Fluxes(),
                         vertical_mixing=GOTM(), tiles="auto", device=DEV)
        dt, depth = 10.0, 100.0
    shape = sim.T.mask.all_values.shape
    wet = sim.T.mask.all_values != 0
    for a in (sim.airsea.taux, sim.airsea.tauy):
        a.all_values.copy_(torch.where(wet, 0.05 + 0.1 * _up(_modes(rng, *shape)), a.all_values))
    zc = sim.T.zc.all_values
    warm = torch.exp(zc / (0.2 * depth))
    t = 4.0 + 16.0 * (zc + depth) / depth + _up(_modes(rng, *shape)) * warm
    s = 35.0 + 0.5 * _up(_modes(rng, *shape)) * warm
    sim.temp.all_values.copy_(torch.where(wet, t, sim.temp.all_values))
    sim.salt.all_values.copy_(torch.where(wet, s, sim.salt.all_values))
    sim.start(dt, case["split"])
    return sim


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    k = case["kind"]
    if k == "step":
        sim = _step_sim(case, seed)
        for a in [sim.T.z, sim.T.hn, sim.momentum.ww] + sim.tracers._tracers:
            a.all_values.masked_fill_(sim.T.land, 0.0)
        runner = DomainRunner(sim)
        runner.prepare()
        return dict(kind=k, runner=runner)
    if k == "transport":
        autotune.apply(None)
        wl = workloads.tracer_transport(nx=case["nx"], ny=case["ny"], nz=case["nz"], seed=seed)
        sim = TracerTransport(wl, device=DEV)
        sim.tracers[0].all_values.masked_fill_(sim.T.land, 0.0)
        return dict(kind=k, sim=sim)
    nz = case.get("nz", 0)
    form = case.get("form", "fp64")
    field = torch.float32 if form == "f32" else F64
    other = F64 if form == "fp64" else torch.float32
    T = _grid(rng, case["nx"], case["ny"], nz, zoom=1.0)
    if k == "adv2d":
        u, v, _ = _flow(T, rng, 1)
        return dict(kind=k, T=T, dt=60.0, u=Array(T.ugrid, u[0].contiguous()), v=Array(T.vgrid, v[0].contiguous()),
                    var=Array(T, _tracer(T, rng, 1, F64)[0].contiguous()),
                    adv=Advection(T, AdvectionScheme(case["scheme"]), AdvectionSplit(case["split"])))
    if k == "adv3d":
        u, v, w = _flow(T, rng, nz)
        ah = [None, None]
        if case["diffusion"]:
            ah = [Array(g, 20.0 + 10.0 * _up(_modes(rng, *T.mask.all_values.shape))) for g in (T.ugrid, T.vgrid)]
        return dict(kind=k, T=T, dt=120.0, u=Array(T.ugrid, u.to(other), z=CENTERS),
                    v=Array(T.vgrid, v.to(other), z=CENTERS), w=Array(T, w.to(other), z=INTERFACES), ah=ah,
                    vars=[Array(T, _tracer(T, rng, nz, field), z=CENTERS) for _ in range(case["nt"])],
                    adv=Advection(T, AdvectionScheme(case["scheme"])))
    shape = T.mask.all_values.shape
    if k == "vdiff":
        s = torch.arange(nz + 1, device=DEV, dtype=F64)[:, None, None] / nz
        nuh = (1e-5 + 4e-2 * s * (1.0 - s) * torch.exp(_up(_modes(rng, *shape)))).to(other)
        T.ho.all_values.mul_(_up(1.0 + 0.01 * _modes(rng, *shape)))
        ea2 = ea4 = None
        if case["sources"]:  # a drag in the bottom layer, a forcing everywhere
            ea2, ea4 = [], []
            for _ in range(case["nt"]):
                a = torch.zeros((nz,) + tuple(shape), dtype=other, device=DEV)
                a[0] = -0.05 * (1.1 + _up(_modes(rng, *shape)))
                ea2.append(Array(T, a, z=CENTERS))
                ea4.append(Array(T, (1e-3 * _up(_modes(rng, *shape)) * (0.5 + s[1:])).to(other), z=CENTERS))
        return dict(kind=k, T=T, dt=120.0, nuh=Array(T, nuh, z=INTERFACES), ea2=ea2, ea4=ea4,
                    vars=[Array(T, _tracer(T, rng, nz, field), z=CENTERS) for _ in range(case["nt"])],
                    mol=[1.4e-7 / (1 + n) for n in range(case["nt"])], vd=VerticalDiffusion(T, cnpar=case["cnpar"]))
    assert k == "ip"
    T.zin = Array(T, 0.3 * _up(_modes(rng, *shape)))
    b = 2e-3 * (_tracer(T, rng, nz, F64) - 12.0)
    b = torch.where(T.mask.all_values != 0, b, 0.0)
    return dict(kind=k, T=T, form=form, buoy=Array(T, b, z=CENTERS), x=T.ugrid.array(z=CENTERS, fill=0.0),
                y=T.vgrid.array(z=CENTERS, fill=0.0), work=torch.zeros((nz + 2,) + tuple(shape), dtype=F64, device=DEV))


def run(st):
    k = st["kind"]
    if k == "step":
        st["runner"].step()
        sim = st["runner"].sim
        m = sim.momentum
        out = dict(z=sim.T.z, U=m.U, V=m.V, uk=m.uk, vk=m.vk, ww=m.ww, hn=sim.T.hn)
        out.update({"t%02d" % n: t for n, t in enumerate(sim.tracers._tracers)})
        return {n: a.all_values for n, a in out.items()}
    if k == "transport":
        st["sim"].step()
        return st["sim"].tracers[0].all_values
    if k == "adv2d":
        st["adv"](st["u"], st["v"], st["dt"], st["var"])
        return dict(var=st["var"].all_values, D=st["adv"].D)
    if k == "adv3d":
        st["adv"].apply_3d_batch(st["u"], st["v"], st["w"], st["dt"], st["vars"], Ah_u=st["ah"][0], Ah_v=st["ah"][1])
        return dict(vars=[v.all_values for v in st["vars"]], h=st["adv"].h)
    if k == "vdiff":
        st["vd"].batch(st["nuh"], st["dt"], st["vars"], st["mol"], st["ea2"], st["ea4"], use_ho=True)
        return [v.all_values for v in st["vars"]]
    _pygetm.shchepetkin_mcwilliams(st["buoy"], st["x"], st["y"], st["work"],
                                   "float32" if st["form"] == "mixed" else "float64")
    return [st["x"].all_values, st["y"].all_values]


def work(case):
    k, n2 = case["kind"], case["nx"] * case["ny"]
    n3, nt = n2 * case.get("nz", 1), case.get("nt", 1)
    field = 4 if case.get("form") == "f32" else 8
    other = 8 if case.get("form", "fp64") == "fp64" else 4
    if k == "adv2d":  # u, v, D on three grids and the field read; the field and D written
        return dict(bytes=8 * 8 * n2, flops=60 * n2)
    if k == "adv3d":  # u, v, w, three thicknesses, the fields; the fields and the thickness written
        return dict(bytes=n3 * (3 * other + 4 * 8 + 2 * field * nt), flops=n3 * (30 + 70 * nt))
    if k == "vdiff":  # nuh, two thicknesses, sources, the fields; the fields written
        return dict(bytes=n3 * (other + 16 + nt * (2 * field + (2 * other if case["sources"] else 0))),
                    flops=n3 * 25 * nt)
    if k == "ip":  # buoyancy, heights, thicknesses; two gradients
        return dict(bytes=n3 * 40, flops=n3 * 90)
    if k == "transport":
        return dict(bytes=n3 * (4 * 8 + 3 * 8 + 16), flops=n3 * 125)
    # a 3D step: velocities, transports, thickness and tracers in and out,
    # and per substep some twenty fields of one plane
    return dict(bytes=2 * n3 * (4 * other + 8 + 8 * nt) + case["split"] * n2 * 8 * 20,
                flops=n3 * (300 + 120 * nt) + case["split"] * n2 * 200)


# ---------------------------------------------------------------------------
# the operators in 64 bits, plainly
# ---------------------------------------------------------------------------
def _limiter(scheme, r, c):
    one = torch.ones_like(r)
    if scheme == 1:
        kap = 1.0 - c
        x = 0.25 * (kap - 1.0 / 3.0 / kap)
        lin = ((0.5 + x) + (0.5 - x) * r).clamp(min=0.0)
        return torch.minimum(torch.minimum(2.0 * r, lin), 2.0 * one)
    if scheme == 2:
        return torch.minimum(torch.minimum(2.0 * r, 0.5 * (1.0 + r)), 2.0 * one)
    if scheme == 3:
        x = (1.0 - 2.0 * c) / 6.0
        lin = (0.5 + x) + (0.5 - x) * r
        return torch.minimum(torch.minimum(2.0 * r / (c + 1e-10), lin), 2.0 / (1.0 - c))
    if scheme == 4:
        return torch.minimum(torch.minimum(2.0 * r, torch.maximum(1.0 + 2.0 * r, 2.0 + r) / 3.0), 2.0 * one)
    if scheme == 5:
        return torch.maximum(torch.minimum(2.0 * r, one), torch.minimum(r, 2.0 * one))
    return torch.zeros_like(r)


def _face(scheme, fuu, fu, fd, c):
    d, du = fd - fu, fu - fuu
    on = d * du > 0
    r = torch.where(on, du / torch.where(on, d, 1.0), 0.0)
    return torch.where(on, fu + 0.5 * _limiter(scheme, r, c) * (1.0 - c) * d, fu)


def _hpass(T, axis, scheme, dt, h, fs, vel, hv, ah):
    """One directional pass over the fields fs (each [k, j, i]); returns the new h and fields."""
    g = T.ugrid if axis == 2 else T.vgrid
    length, inv = (g.dy, g.idx) if axis == 2 else (g.dx, g.idy)
    m = _wet(g)
    ny, nx = m.shape
    inside = torch.zeros_like(m)
    x0, y0 = T.halox, T.haloy
    if axis == 2:
        inside[y0:y0 + T.ny, x0 - 1:x0 + T.nx] = True
    else:
        inside[y0 - 1:y0 + T.ny, x0:x0 + T.nx] = True
    cells = torch.zeros_like(m)
    cells[y0:y0 + T.ny, x0:x0 + T.nx] = True
    cells &= T.mask.all_values == 1
    act = m & inside
    q = torch.where(act, vel * torch.where(act, hv, 0.0) * length.all_values, 0.0)
    c = torch.where(act, (vel * dt * inv.all_values).abs(), 0.0)
    up = vel > 0
    sh = lambda a, n: torch.roll(a, -n, dims=axis - 3 if a.dim() == 2 else axis)  # noqa: E731  (wraps only where inactive)
    low = lambda a: torch.roll(a, 1, dims=axis)  # noqa: E731
    iA = T.iarea.all_values
    hnew = torch.where(cells, h - dt * (q - low(q)) * iA, h)
    mw, me = sh(m, -1), sh(m, 1)
    out = []
    for f in fs:
        fm, f1, f2 = sh(f, -1), sh(f, 1), sh(f, 2)
        fu, fd = torch.where(up, f, f1), torch.where(up, f1, f)
        fuu = torch.where(up, torch.where(mw, fm, f), torch.where(me, f2, f1))
        flux = torch.where(act, q * _face(scheme, fuu, fu, fd, c), 0.0)
        if ah is not None:
            flux = flux - torch.where(act, ah * torch.where(act, hv, 0.0) * (f1 - f) * inv.all_values * length.all_values,
                                      0.0)
        out.append(torch.where(cells, (h * f - dt * ((flux - low(flux)) * iA)) / torch.where(cells, hnew, 1.0), f))
    return hnew, out


def _wpass(T, scheme, dt, h, f, w):
    """Vertical pass of one field with the column-wise sub-steps."""
    nz = f.shape[0]
    cells = torch.zeros_like(T.mask.all_values, dtype=torch.bool)
    cells[T.haloy:T.haloy + T.ny, T.halox:T.halox + T.nx] = True
    cells &= T.mask.all_values == 1
    h0, f0, w = h[:, cells], f[:, cells], w[:, cells]
    hc, fc = h0, f0
    iters = torch.ones(h0.shape[1], device=f.device, dtype=F64)
    it = torch.ones_like(iters)
    while bool((it <= iters).any()) and nz > 1:
        cfl = (w[1:-1].abs() * dt / torch.minimum(hc[:-1], hc[1:])).amax(0)
        need = torch.where(cfl > 1.0, cfl.ceil(), 1.0).clamp(max=200.0)
        grow = (need > iters) & (it <= iters)
        iters = torch.where(grow, need, iters)
        back = grow & (it > 1)
        hc, fc = torch.where(back, h0, hc), torch.where(back, f0, fc)
        it = torch.where(back, 1.0, it)
        wi = w[1:-1]
        c = wi.abs() * dt / torch.minimum(hc[:-1], hc[1:]) / iters
        below = torch.cat([fc[:1], fc[:-2]])
        above = torch.cat([fc[2:], fc[-1:]])
        up = wi > 0
        fu, fd = torch.where(up, fc[:-1], fc[1:]), torch.where(up, fc[1:], fc[:-1])
        flux = wi * _face(scheme, torch.where(up, below, above), fu, fd, c)
        z = torch.zeros_like(flux[:1])
        flux = torch.cat([z, flux, z])
        d = dt / iters
        hn = hc - d * (w[1:] - w[:-1])
        fn = (hc * fc - d * (flux[1:] - flux[:-1])) / hn
        go = it <= iters
        hc, fc = torch.where(go, hn, hc), torch.where(go, fn, fc)
        it = it + go
    hout, fout = h.clone(), f.clone()
    hout[:, cells], fout[:, cells] = hc, fc
    return hout, fout


def _advect(T, scheme, dt, h, fs, u, v, w, ah, ufirst):
    order = [2, 1] if ufirst else [1, 2]
    vel, hv, a = {2: u, 1: v}, {2: T.ugrid.hn.all_values, 1: T.vgrid.hn.all_values}, {2: ah[0], 1: ah[1]}
    for ax in order:
        h, fs = _hpass(T, ax, scheme, 0.5 * dt, h, fs, vel[ax], hv[ax], a[ax])
    pairs = [_wpass(T, scheme, dt, h, f, w) for f in fs]
    h, fs = pairs[-1][0], [p[1] for p in pairs]
    for ax in reversed(order):
        h, fs = _hpass(T, ax, scheme, 0.5 * dt, h, fs, vel[ax], hv[ax], a[ax])
    return h, fs


def _diffuse(mask, nuh, dt, cnpar, mol, ho, hn, f, ea2, ea4):
    nz = f.shape[0]
    wet = mask == 1
    nuh, ho, hn, x = nuh[:, wet], ho[:, wet], hn[:, wet], f[:, wet]
    a = 2.0 * dt * (nuh[1:-1] + mol)
    ao, an = (1.0 - cnpar) * a / (ho[1:] + ho[:-1]), cnpar * a / (hn[1:] + hn[:-1])
    z = torch.zeros_like(x[:1])
    up, lo = torch.cat([an, z]), torch.cat([z, an])
    diag = hn + up + lo
    d = torch.cat([ao * (x[1:] - x[:-1]), z])
    rhs = x * ho + d - torch.cat([z, ao * (x[1:] - x[:-1])])
    if ea2 is not None:
        diag = diag - ea2[:, wet]
    if ea4 is not None:
        rhs = rhs + ea4[:, wet]
    r, q = torch.empty_like(x), torch.empty_like(x)
    r[nz - 1], q[nz - 1] = lo[nz - 1] / diag[nz - 1], rhs[nz - 1] / diag[nz - 1]
    for k in range(nz - 2, -1, -1):  # x_k = q_k + r_k x_{k-1}
        den = diag[k] - up[k] * r[k + 1]
        r[k], q[k] = lo[k] / den, (rhs[k] + up[k] * q[k + 1]) / den
    new = torch.empty_like(x)
    new[0] = q[0]
    for k in range(1, nz):
        new[k] = q[k] + r[k] * new[k - 1]
    out = f.clone()
    out[:, wet] = new
    return out


def _harm(a, b, eps=1e-10):
    p = 2.0 * a * b
    on = p > eps
    return torch.where(on, p / torch.where(on, a + b, 1.0), 0.0)


def _pressure(T, b):
    """Shchepetkin and McWilliams (2003) density-Jacobian pressure gradients."""
    nz = b.shape[0]
    h, zc, z = T.hn.all_values, T.zc.all_values, T.zin.all_values
    x = 1.0 / 12.0
    dr, dz = b[1:] - b[:-1], zc[1:] - zc[:-1]
    dr, dz = torch.cat([dr[:1], dr, dr[-1:]]), torch.cat([dz[:1], dz, dz[-1:]])
    hr = _harm(dr[1:], dr[:-1])
    sz = dz[1:] + dz[:-1]
    hz = torch.where(sz != 0, 2.0 * dz[1:] * dz[:-1] / torch.where(sz != 0, sz, 1.0), 0.0)
    dr, dz = dr[1:-1], dz[1:-1]
    part = 0.5 * ((b[1:] + b[:-1]) * dz - 0.2 * ((hr[1:] - hr[:-1]) * (dz - x * (hz[1:] + hz[:-1]))
                                                 - (hz[1:] - hz[:-1]) * (dr - x * (hr[1:] + hr[:-1]))))
    top = (b[-1] + 0.5 * dr[-1] * 0.5 * h[-1] / torch.where(dz[-1] != 0, dz[-1], 1.0)) * 0.5 * h[-1]
    P = torch.cat([top[None] + part.flip(0).cumsum(0).flip(0), top[None]])
    out = []
    for axis, g, inv in ((2, T.ugrid, T.ugrid.idx), (1, T.vgrid, T.vgrid.idy)):
        m = g.mask.all_values
        sh = lambda a, n: torch.roll(a, -n, dims=axis - 3 if a.dim() == 2 else axis)  # noqa: E731
        rz, rr = torch.where(m > 0, sh(zc, 1) - zc, 0.0), torch.where(m > 0, sh(b, 1) - b, 0.0)
        z0, z1 = _harm(sh(rz, -1), rz), _harm(rz, sh(rz, 1))
        r0, r1 = _harm(sh(rr, -1), rr), _harm(rr, sh(rr, 1))
        fc = 0.5 * ((sh(b, 1) + b) * rz - 0.2 * ((r1 - r0) * (rz - x * (z1 + z0)) - (z1 - z0) * (rr - x * (r1 + r0))))
        surf = (sh(z, 1) - z) * 0.5 * (sh(b[-1], 1) + b[-1])
        val = 0.5 * (h + sh(h, 1)) * inv.all_values * (sh(P, 1) - P + fc - surf)
        on = torch.zeros_like(m, dtype=torch.bool)
        on[T.haloy:T.haloy + T.ny, T.halox:T.halox + T.nx] = True
        out.append(torch.where(on & (m == 1), val, 0.0))
    return out


def exact(case, seed):
    k = case["kind"]
    if k == "step":  # a whole model: its single layers are the cases above
        return None
    st = prepare(case, seed)
    if k == "transport":
        s = st["sim"]
        T, f = s.T, s.tracers[0].all_values.clone()
        _, (f,) = _advect(T, 5, s.dt, T.ho.all_values, [f], s.uk.all_values, s.vk.all_values, s.w.all_values,
                          (None, None), False)
        return _diffuse(T.mask.all_values, s.nuh.all_values, s.dt, 1.0, 0.0, T.hn.all_values, T.hn.all_values, f, None,
                        None)
    T = st["T"]
    if k == "adv2d":
        h, f = T.D.all_values[None], [st["var"].all_values[None].clone()]
        vel = {2: st["u"].all_values[None], 1: st["v"].all_values[None]}
        hv = {2: T.ugrid.D.all_values[None], 1: T.vgrid.D.all_values[None]}
        dt = st["dt"]
        seq = {1: [(1, dt), (2, dt)], 2: [(1, dt / 2), (2, dt), (1, dt / 2)],
               3: [(1, dt / 2), (2, dt / 2), (2, dt / 2), (1, dt / 2)]}[case["split"]]
        for ax, d in seq:
            h, f = _hpass(T, ax, case["scheme"], d, h, f, vel[ax], hv[ax], None)
        return dict(var=f[0][0], D=h[0])
    if k == "adv3d":
        ah = tuple(None if a is None else a.all_values for a in st["ah"])
        h, f = _advect(T, case["scheme"], st["dt"], T.ho.all_values, [v.all_values.to(F64) for v in st["vars"]],
                       st["u"].all_values.to(F64), st["v"].all_values.to(F64), st["w"].all_values.to(F64), ah, False)
        return dict(vars=f, h=h)
    if k == "vdiff":
        wide = lambda a, n: None if a is None else a[n].all_values.to(F64)  # noqa: E731
        return [_diffuse(T.mask.all_values, st["nuh"].all_values.to(F64), st["dt"], case["cnpar"], st["mol"][n],
                         T.ho.all_values, T.hn.all_values, v.all_values.to(F64), wide(st["ea2"], n), wide(st["ea4"], n))
                for n, v in enumerate(st["vars"])]
    return _pressure(T, st["buoy"].all_values)
