"""The workloads by which the speed of the engine is measured.

Each case is a call, or the few calls that belong together, that a program
using this package makes over and over: one travel-time solve and its adjoint
(the drop-in for the reference's solver), a batch of events, one misfit
gradient, receiver times with their autograd gradient, dispersion with its
depth kernels, kernel smoothing, one optimiser step and the topography media.
Sizes follow the package's own configurations (``workloads.py``: 41x41x30 at
0.05 deg up to 301x301x40 at 0.01 deg and 601x601x50 at 0.005 deg) and ragged
sizes between them.

Inputs are seeded: a gradient model (2.8-4.6 km/s) with a Gaussian random
field of +-6 %, stations at random places as sources and receivers, observed
times from straight rays with 2 % noise, fractal topography of 4 km relief.

``exact`` restates a path in plain torch, FP64, where that takes seconds: the
sweeps by anti-diagonals (each cell reads its axis neighbours only, so that
is the raster order of the Gauss-Seidel sweeps), the smoothing steps, the
two-loop recursion and the topography media.
"""
from __future__ import annotations

import math

import numpy as np
import torch

R = 6371.0
RAD = math.pi / 180.0
DEV = "cuda"
F64 = dict(dtype=torch.float64, device=DEV)


def listed():
    return [
        # one source through the solver's host interface, as the reference's
        # callers use it: the example's grid, and a large one on topography
        dict(name="solve-41x41", kind="solve", nx=41, ny=41, step=0.05, topo=False, nsta=25,
             precision="fp64"),
        dict(name="solve-301x251-topo", kind="solve", nx=301, ny=251, step=0.01, topo=True,
             nsta=100, precision="fp64"),
        # one misfit gradient of an inversion: the checkerboard example (25
        # stations, FP64) and the dense-array batch (8000 solves, FP32 sweeps)
        dict(name="gradient-41x41x30", kind="gradient", nx=41, ny=41, nz=30, step=0.05, nper=10,
             pmin=4.0, pmax=40.0, nsta=25, precision="fp64"),
        dict(name="gradient-301x301x40", kind="gradient", nx=301, ny=301, nz=40, step=0.01,
             nper=20, pmin=2.0, pmax=50.0, nsta=400, precision="fp32"),
        # event batches with given phase velocities: an uneven batch on
        # topography (about 40 receivers an event), and a regional FP64 one
        dict(name="events-201x201-topo", kind="events", nx=201, ny=201, step=0.01, nper=15,
             pmin=4.0, pmax=40.0, nsta=310, nrec=40, topo=True, precision="fp32"),
        dict(name="events-151x137", kind="events", nx=151, ny=137, step=0.02, nper=12, pmin=3.0,
             pmax=40.0, nsta=100, nrec=0, topo=False, precision="fp64"),
        # receiver times and the exact gradient of a loss on them, by autograd
        dict(name="traveltimes-61x53x25", kind="traveltimes", nx=61, ny=53, nz=25, step=0.04,
             nper=8, pmin=4.0, pmax=32.0, nsta=16, convention="exact", precision="fp64"),
        # group velocities and their depth kernels of a regional model
        dict(name="columns-101x87x33-group", kind="columns", nx=101, ny=87, nz=33, step=0.02,
             nper=12, pmin=3.0, pmax=40.0, wave="rayleigh", data="group"),
        # kernel smoothing after a gradient: the example's grid and the largest
        dict(name="smooth-41x41x30", kind="smooth", nx=41, ny=41, nz=30, step=0.05, sigma_h=0.2,
             sigma_v=6.0),
        dict(name="smooth-601x601x50", kind="smooth", nx=601, ny=601, nz=50, step=0.005,
             sigma_h=0.025, sigma_v=6.0),
        # one optimiser step: history, L-BFGS direction, its angle, the update
        dict(name="lbfgs-301x301x40", kind="lbfgs", nx=301, ny=301, nz=40, history=5),
        # the media of a surface with topography, smoothed per period
        dict(name="topography-201x201", kind="topography", nx=201, ny=201, step=0.01, nper=15,
             pmin=4.0, pmax=40.0),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve", "solve", "gradient", "events", "events", "traveltimes", "columns",
                       "columns", "smooth", "smooth", "lbfgs", "topography"])
    if kind == "lbfgs":
        return dict(kind=kind, nx=size(31, 401), ny=size(31, 401), nz=rng.randint(15, 50),
                    history=rng.randint(1, 5))
    nx = size(31, 301)
    ny = max(27, min(320, int(nx * rng.uniform(0.7, 1.4))))
    c = dict(kind=kind, nx=nx, ny=ny, step=round(2.5 / max(nx, ny), 5))
    if kind == "smooth":
        sh, sv = rng.uniform(2.0, 6.0) * c["step"], round(rng.uniform(2.0, 9.0), 2)
        return dict(c, nz=rng.randint(15, 50), sigma_h=round(sh, 5), sigma_v=sv)
    if kind == "solve":
        return dict(c, topo=rng.random() < 0.5, nsta=size(5, 200),
                    precision=rng.choice(["fp64", "fp64", "fp32"]))
    nper = rng.randint(4, 18)
    c.update(nper=nper, pmin=round(rng.uniform(2.0, 5.0), 2), pmax=round(rng.uniform(25.0, 50.0), 2))
    if kind == "topography":
        return dict(c, nx=min(nx, 221), ny=min(ny, 221), nper=min(nper, 15))
    if kind == "columns":
        wave, data = rng.choice([("rayleigh", "phase"), ("rayleigh", "group"), ("love", "phase"),
                                 ("love", "group")])
        top = 120 if data == "group" else 200
        return dict(c, nx=min(nx, top), ny=min(ny, top), nz=rng.randint(15, 45), wave=wave,
                    data=data)
    precision = rng.choice(["fp64", "fp32"])
    # cell updates of the batch, the FP64 ones counted four times, stay below
    # half the largest listed batch
    most = 3.0e8 / (nx * ny * nper * (4 if precision == "fp64" else 1))
    nsta = max(4, min(size(8, 300), int(most)))
    if kind == "events":
        return dict(c, nsta=nsta, nrec=rng.choice([0, 10, 40]), topo=rng.random() < 0.4,
                    precision=precision)
    if kind == "gradient":
        return dict(c, nz=rng.randint(15, 45), nsta=nsta, precision=precision)
    convention = rng.choice(["reference", "derivative", "exact"])
    return dict(c, nx=min(nx, 120), ny=min(ny, 120), nz=rng.randint(15, 40), nsta=min(nsta, 40),
                convention=convention, precision="fp64" if convention == "exact" else precision)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _grid(c):
    return 102.0 + c["step"] * np.arange(c["nx"]), 24.0 + c["step"] * np.arange(c["ny"])


def _depths(c):
    return 2.0 * np.arange(c["nz"])


def _periods(c):
    return np.geomspace(c["pmin"], c["pmax"], c["nper"])


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _field(g, shape, spacing, corr):
    """Gaussian random field of unit deviation: filtered white noise."""
    w = torch.fft.fftn(torch.randn(shape, generator=g, **F64))
    k2 = 0.0
    for i, (n, d) in enumerate(zip(shape, spacing)):
        k = torch.fft.fftfreq(n, d=d, **F64) ** 2
        k2 = k2 + k.reshape([-1 if j == i else 1 for j in range(len(shape))])
    f = torch.fft.ifftn(w * torch.exp(-0.5 * (2 * math.pi * corr) ** 2 * k2)).real
    return f / f.std()


def _model(c, seed):
    """vs (nx, ny, nz): the gradient model with the random field."""
    z = torch.as_tensor(_depths(c), **F64)
    km = c["step"] * RAD * R
    f = _field(_gen(seed), (c["nx"], c["ny"], c["nz"]), (km, km, 2.0), 15.0)
    vs = (2.8 + 1.8 * z / z[-1]) * (1.0 + 0.06 * torch.clamp(f / 2.0, -1.0, 1.0))
    return vs.contiguous()


def _velocities(c, seed):
    """Phase velocities (nper, ny, nx): rising with the period, +-5 %."""
    km = c["step"] * RAD * R
    f = _field(_gen(seed), (c["nper"], c["ny"], c["nx"]), (4.0, km, km), 20.0)
    return (_reference(c)[:, None, None] * (1.0 + 0.05 * torch.clamp(f / 2.0, -1.0, 1.0))).contiguous()


def _reference(c):
    lp = torch.log(torch.as_tensor(_periods(c), **F64))
    return 2.9 + 0.9 * (lp - lp[0]) / (lp[-1] - lp[0])


def _slopes(c, seed, nper):
    """Media (nper, ny, nx) of a smooth fractal surface: m11, m12, m22."""
    g = _gen(seed + 7)
    km = c["step"] * RAD * R
    z = _field(g, (c["ny"], c["nx"]), (km, km), 6.0)
    out = [[], [], []]
    for ip in range(nper):
        h = z * (1.2 / (1.0 + 0.3 * ip))
        fy, fx = torch.gradient(h, spacing=km)
        den = 1.0 + fx * fx + fy * fy
        for o, v in zip(out, ((1.0 + fy * fy) / den, -(fx * fy / den), (1.0 + fx * fx) / den)):
            o.append(v)
    return [torch.stack(o).contiguous() for o in out]


def _stations(c, rng):
    xx, yy = _grid(c)
    s = c["step"]
    return (rng.uniform(xx[0] + 2 * s, xx[-1] - 2 * s, c["nsta"]),
            rng.uniform(yy[0] + 2 * s, yy[-1] - 2 * s, c["nsta"]))


def _events(c, seed):
    """Events of (source, period) pairs with observed straight-ray times: all
    other stations as receivers (nrec 0) or Poisson(nrec) of them, and then a
    random set of sources for each period."""
    rng = np.random.default_rng(seed)
    n, nper = c["nsta"], c["nper"]
    lo, la = _stations(c, rng)
    r = RAD
    dist = np.arccos(np.clip(np.sin(la[:, None] * r) * np.sin(la * r) + np.cos(la[:, None] * r)
                             * np.cos(la * r) * np.cos((lo[:, None] - lo) * r), -1, 1)) * R
    if not c.get("nrec"):
        src = np.repeat(np.arange(n), nper)
        iper = np.tile(np.arange(nper, dtype=np.int32), n)
        k = np.tile(np.arange(n - 1), n * nper)
        idx = k + (k >= np.repeat(src, n - 1))
        cnt = np.full(n * nper, n - 1)
    else:
        src, iper, idx, cnt = [], [], [], []
        counts = np.random.default_rng(n)     # how many is the case's, which the seed's
        for ip in range(nper):
            for s in rng.choice(n, size=counts.integers(max(1, n // 6), n + 1), replace=False):
                k = max(1, min(n - 1, counts.poisson(c["nrec"])))
                rec = np.sort(rng.permutation(n - 1)[:k])
                src.append(s)
                iper.append(ip)
                idx.append(rec + (rec >= s))
                cnt.append(k)
        src, iper, idx = np.array(src), np.array(iper, np.int32), np.concatenate(idx)
    ptr = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32)
    cref = _reference(c).cpu().numpy()
    tt = dist[np.repeat(src, cnt), idx] / cref[np.repeat(iper, cnt)]
    tt = tt * (1.0 + 0.02 * rng.standard_normal(tt.size))
    return dict(evlo=lo[src], evla=la[src], iper=iper, rec_ptr=ptr, rec_idx=idx.astype(np.int32),
                stlo=lo, stla=la), tt


def _plan(c, seed):
    from surfattpp_b200 import preproc
    ev, tt = _events(c, seed)
    plan = preproc.ForwardAdjointPlan(*_grid(c), c["nper"], ev["evlo"], ev["evla"], ev["iper"],
                                      ev["rec_ptr"], ev["rec_idx"], ev["stlo"], ev["stla"],
                                      precision=c["precision"])
    return plan, torch.as_tensor(tt, **F64), torch.ones(tt.size, **F64)


def _solve_inputs(c, seed):
    rng = np.random.default_rng(seed)
    xx, yy = _grid(c)
    one = dict(c, nper=2, pmin=10.0, pmax=20.0)
    fun = (1.0 / _velocities(one, seed)[0]).cpu().numpy()
    if c["topo"]:
        m11, m12, m22 = (m[0].cpu().numpy() for m in _slopes(c, seed, 1))
    else:
        m11, m12, m22 = np.ones(fun.shape), np.zeros(fun.shape), np.ones(fun.shape)
    lo, la = _stations(c, rng)
    return dict(xx=xx, yy=yy, spha=m11, sphb=m22, sphc=-m12, fun=fun, x0=lo[0], y0=la[0],
                xrec=lo[1:], yrec=la[1:], src=rng.normal(0.0, 1.0, c["nsta"] - 1))


def _kernel(c, seed):
    """A sensitivity kernel (nx, ny, nz): rough over cells, decaying with depth."""
    g = _gen(seed)
    k = torch.randn((c["nx"], c["ny"], c["nz"]), generator=g, **F64)
    return (k * torch.exp(-torch.arange(c["nz"], **F64) / 12.0)).contiguous()


def _iterates(c, seed):
    """Models and gradients of `history` + 1 iterations that converge slowly."""
    n = c["nx"] * c["ny"] * c["nz"]
    g = _gen(seed)
    target = 3.5 + 0.3 * torch.randn(n, generator=g, **F64)
    scale = 0.5 + torch.rand(n, generator=g, **F64)
    m, out = torch.full((n,), 3.5, **F64), []
    for _ in range(c["history"] + 1):
        grad = scale * (m - target) / 50.0
        out.append((m.clone(), grad))
        m = m * (1.0 - 0.02 * grad / grad.abs().max())
    return out


def _surface(c, seed):
    """Raw topography (km, 0 to 4) on a margin around the grid, power ~ 1/k^2,
    and the smoothing width of each period (2.5 wavelengths over 2 pi)."""
    xx, yy = _grid(c)
    lon = np.arange(xx[0] - 0.2, xx[-1] + 0.2 + 1e-9, 0.005)
    lat = np.arange(yy[0] - 0.2, yy[-1] + 0.2 + 1e-9, 0.005)
    w = np.fft.fft2(np.random.default_rng(seed).standard_normal((lat.size, lon.size)))
    k = np.hypot(np.fft.fftfreq(lat.size)[:, None], np.fft.fftfreq(lon.size)[None, :])
    k[0, 0] = np.inf
    z = np.fft.ifft2(w / k).real
    z = 4.0 * (z - z.min()) / (z.max() - z.min())
    sig = _reference(c).cpu().numpy() * _periods(c) * 2.5 / (2.0 * math.pi) / (R * RAD)
    return dict(xx=xx, yy=yy, lon=lon, lat=lat, z=z, sig=sig)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "solve":
        return dict(c=c, **_solve_inputs(c, seed))
    if kind == "events":
        plan, tt, wt = _plan(c, seed)
        m = _slopes(c, seed, c["nper"]) if c["topo"] else [None] * 3
        return dict(c=c, plan=plan, svel=_velocities(c, seed), tt=tt, wt=wt, media=m, out={})
    if kind in ("gradient", "traveltimes"):
        from surfattpp_b200 import inversion
        plan, tt, wt = _plan(c, seed)
        if c.get("convention") == "exact":
            plan.set_adjoint("exact")
        grad = inversion.MisfitGradient(plan, _depths(c), _periods(c))
        return dict(c=c, grad=grad, vs=_model(c, seed), tt=tt, wt=wt, out={})
    if kind == "columns":
        return dict(c=c, vs=_model(c, seed), z=_depths(c), periods=_periods(c))
    if kind == "smooth":
        return dict(c=c, ker=_kernel(c, seed), y=_grid(c)[1], z=_depths(c))
    if kind == "lbfgs":
        from surfattpp_b200 import optimize
        its = _iterates(c, seed)
        lb = optimize.LBFGS(its[0][0].numel())
        for i, (m, g) in enumerate(its[:-1]):
            lb.store(i, m, g)
        return dict(c=c, lb=lb, model=its[-1][0], grad=its[-1][1])
    return dict(c=c, **_surface(c, seed))


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(s):
    c, kind = s["c"], s["c"]["kind"]
    if kind == "solve":
        from surfattpp_b200 import eikonal
        T, fit = eikonal.FSM_UW_PS_lonlat_2d(s["xx"], s["yy"], s["spha"], s["sphb"], s["sphc"],
                                             s["fun"], s["x0"], s["y0"], c["precision"], True)
        Ta, ait = eikonal.FSM_O1_JSE_lonlat_2d(s["xx"], s["yy"], s["spha"], s["sphb"], s["sphc"], T,
                                               s["xrec"], s["yrec"], s["src"], c["precision"], True)
        return dict(T=T, fit=fit, Ta=Ta, ait=ait)
    if kind == "events":
        return dict(s["plan"].run(s["svel"], s["tt"], s["wt"], True, *s["media"], out=s["out"]))
    if kind == "gradient":
        return dict(s["grad"].run(s["vs"], s["tt"], s["wt"], out=s["out"]))
    if kind == "traveltimes":
        from surfattpp_b200 import inversion
        v = s["vs"].detach().requires_grad_(True)
        T = inversion.TravelTimes.apply(s["grad"], v, c["convention"])
        chi = 0.5 * (s["wt"] * (T - s["tt"]) ** 2).sum()
        (g,) = torch.autograd.grad(chi, v)
        return dict(T=T.detach(), chi=chi.detach(), grad=g)
    if kind == "columns":
        from surfattpp_b200 import surfker
        z, p, vs = s["z"], s["periods"], s["vs"]
        igr = int(c["data"] == "group")
        sv, st = surfker.fwdsurf(z, vs, p, iwave=2 if c["wave"] == "rayleigh" else 1, igr=igr)
        if c["wave"] == "love":
            sen = surfker.depthkernel_love(z, vs, p, igr)
        elif igr:
            sen = surfker.depthkernel_group(z, vs, p)
        else:
            sen = surfker.depthkernel_hti(z, vs, p, sv)
        return dict(svel=sv, status=st, sen=sen)
    if kind == "smooth":
        from surfattpp_b200 import postproc
        return postproc.kernel_smooth([s["ker"]], s["y"], s["z"], c["step"], c["step"], 2.0,
                                      c["sigma_h"], c["sigma_v"])
    if kind == "lbfgs":
        from surfattpp_b200 import optimize
        it = c["history"]
        s["lb"].store(it, s["model"], s["grad"])
        d = s["lb"].direction(it)
        top = optimize.grad_normalization(d)
        angle = optimize.calc_descent_angle(d, s["grad"])
        return dict(dir=d, top=top, angle=angle,
                    model=optimize.model_update_vs(s["model"], d, 0.02))
    from surfattpp_b200 import surfgrid
    zg = surfgrid.grid_topography(s["lon"], s["lat"], s["z"], s["xx"], s["yy"])
    return dict(zg=zg, media=surfgrid.build_media_with_topo(s["xx"], s["yy"], zg, s["sig"]))


def _nstep(c):
    top = min(abs(24.0 + c["step"] * (c["ny"] - 1)), 89.0)
    h = c["step"] ** 2 * math.cos(top * RAD) ** 2 / 6.0
    return max(1, math.ceil(c["sigma_h"] ** 2 / (2 * h)), math.ceil(c["sigma_v"] ** 2 / (8.0 / 6.0)))


def work(case):
    """Bytes: inputs read and outputs written once.  Operations: one
    iteration of four sweeps per solve (100 a forward cell update, 12 an
    adjoint one), 20 evaluations of the secular function per root with 150 a
    layer, 400 a layer for the depth kernels, 21 a smoothing update, 60 a
    point of a topography window."""
    c, kind = case, case["kind"]
    n = c["nx"] * c["ny"]
    if kind == "solve":
        return dict(bytes=8.0 * n * 9, flops=4.0 * 112 * n)
    if kind == "smooth":
        m = n * c["nz"]
        return dict(bytes=16.0 * m, flops=21.0 * m * _nstep(c))
    if kind == "lbfgs":
        m, h = n * c["nz"], c["history"]
        return dict(bytes=8.0 * m * (2 * (h + 1) + 4), flops=m * (14.0 * h + 60.0))
    if kind == "topography":
        sig = _surface(c, 0)["sig"]
        pts = sum(min(2 * int(3 * s / c["step"]) + 1, c["nx"])
                  * min(2 * int(3 * s / 0.9 / c["step"]) + 1, c["ny"]) for s in sig)
        return dict(bytes=8.0 * n * (1 + 4 * c["nper"]), flops=60.0 * n * pts)
    nper = c["nper"]
    b, f = 0.0, 0.0
    if kind != "columns":
        ne = c["nsta"] * nper * (0.58 if c.get("nrec") else 1.0)
        nr = ne * (min(c["nrec"], c["nsta"]) if c.get("nrec") else c["nsta"] - 1)
        b += 8.0 * n * nper * (5 if c.get("topo") else 2) + 28.0 * nr
        f += ne * n * 4.0 * 112
    if kind != "events":
        m = n * c["nz"]
        group = c.get("data") == "group"
        b += 16.0 * m + 8.0 * n * nper + (24.0 * m * nper if kind == "columns" else 0.0)
        f += m * nper * (20 * 150.0 * (5 if group else 1) + 400.0 * (3 if group else 1))
    return dict(bytes=b, flops=f)


# ---------------------------------------------------------------------------
# The same results in plain torch, FP64
# ---------------------------------------------------------------------------
def _tensor(a):
    return torch.as_tensor(np.asarray(a), **F64)


def _diagonals(nx, ny, xd, yd):
    """Cells (flat index) of each anti-diagonal in the sweep's order."""
    ix = torch.arange(nx, device=DEV).repeat(ny)
    iy = torch.arange(ny, device=DEV).repeat_interleave(nx)
    d = (ix if xd > 0 else nx - 1 - ix) + (iy if yd > 0 else ny - 1 - iy)
    order = torch.argsort(d, stable=True)
    return torch.split(order, torch.bincount(d, minlength=nx + ny - 1).tolist())


_DIRS = ((1, 1), (1, -1), (-1, 1), (-1, -1))


def _cell(x, x0, d, n):
    i = torch.clamp(torch.floor((x0 - x[0]) / d), 0, n - 2).long()
    return i, torch.clamp((x0 - x[i]) / d, max=1.0)


def _corners(xx, yy, x0, y0):
    """Flat indices and weights [m, 4] of points on the uniform grid."""
    nx = xx.numel()
    i, r1 = _cell(xx, x0, xx[1] - xx[0], nx)
    j, r2 = _cell(yy, y0, yy[1] - yy[0], yy.numel())
    k = j * nx + i
    return (torch.stack([k, k + nx, k + 1, k + nx + 1], -1),
            torch.stack([(1 - r1) * (1 - r2), (1 - r1) * r2, r1 * (1 - r2), r1 * r2], -1))


def _forward(xx, yy, m, f, x0, y0):
    """Factored fast sweeping of events [ne] with media m = (spha, sphb,
    sphc), each [ne or 1, n], and slowness f [ne, n]: travel times [ne, n]."""
    nx, ny, ne = xx.numel(), yy.numel(), f.shape[0]
    xx, yy, x0, y0 = xx * RAD, yy * RAD, x0 * RAD, y0 * RAD
    dx, dy = xx[1] - xx[0], yy[1] - yy[0]
    X, Y = xx.repeat(ny), yy.repeat_interleave(nx)
    a = m[0] / (R * torch.cos(Y)) ** 2
    b = m[1] / R ** 2
    cc = m[2] / (R * R * torch.cos(Y))
    a, b, cc = (v.expand(ne, -1) for v in (a, b, cc))
    k4, w4 = _corners(xx, yy, x0, y0)
    fun0 = (f.gather(1, k4) * w4).sum(1, keepdim=True)
    x0, y0 = x0[:, None], y0[:, None]
    cosd = torch.clamp(torch.sin(Y) * torch.sin(y0) + torch.cos(Y) * torch.cos(y0)
                       * torch.cos(X - x0), -1, 1)
    sind = torch.sqrt(torch.clamp(1 - cosd * cosd, min=0))
    far = sind >= 1e-14
    sind = torch.where(far, sind, 1.0)
    t0 = torch.acos(cosd) * R * fun0
    t0x = torch.where(far, torch.cos(Y) * torch.cos(y0) * torch.sin(X - x0) / sind * R * fun0, 0.0)
    t0y = torch.where(far, -(torch.cos(Y) * torch.sin(y0) - torch.sin(Y) * torch.cos(y0)
                             * torch.cos(X - x0)) / sind * R * fun0, 0.0)
    free = ~(((X - x0).abs() / dx <= 1) & ((Y - y0).abs() / dy <= 1))
    tau = torch.where(free, 10.0, 1.0).to(torch.float64)
    ix = torch.arange(nx, device=DEV).repeat(ny)
    iy = torch.arange(ny, device=DEV).repeat_interleave(nx)
    plans = [[] for _ in _DIRS]
    step = torch.tensor([-1, 1, -nx, nx], device=DEV)[:, None]
    for s, (xd, yd) in enumerate(_DIRS):
        for k in _diagonals(nx, ny, xd, yd):
            has = torch.stack([ix[k] > 0, ix[k] < nx - 1, iy[k] > 0, iy[k] < ny - 1])
            plans[s].append((k, torch.where(has, k + step, k), has))
    sx, sy = (torch.tensor(v, **F64).reshape(4, 1, 1) for v in ((-1, -1, 1, 1), (-1, 1, -1, 1)))
    qx_, qy_ = torch.tensor([0, 0, 1, 1], device=DEV), torch.tensor([2, 3, 2, 3], device=DEV)
    sa = torch.tensor([-1.0, 1.0, -1.0, 1.0], **F64).reshape(4, 1, 1)
    pm = torch.tensor([1.0, -1.0], **F64).reshape(2, 1, 1, 1)
    inf = torch.tensor(math.inf, **F64)
    act = torch.arange(ne, device=DEV)
    T, iters = torch.empty_like(tau), 0
    v = [tau, t0, t0x, t0y, a, b, cc, f, free]
    while act.numel() and iters < 2000:
        iters += 1
        tau, t0, t0x, t0y, a, b, cc, f, free = v
        old = tau.clone()
        for plan in plans:
            for k, kn, has in plan:
                tk, A, B, C, F = t0[:, k], a[:, k], b[:, k], cc[:, k], f[:, k]
                gx, gy = t0x[:, k], t0y[:, k]
                tn = tau[:, kn].transpose(0, 1)          # [4, ne, L]: x-, x+, y-, y+
                tx, ty = tk / dx, tk / dy
                px, qx = gx - sx * tx, sx * tx * tn[qx_]
                py, qy = gy - sy * ty, sy * ty * tn[qy_]
                ea = A * px * px + B * py * py - 2 * C * px * py
                eb = 2 * (A * px * qx + B * py * qy - C * (px * qy + py * qx))
                ec = A * qx * qx + B * qy * qy - 2 * C * qx * qy - F * F
                D = eb * eb - 4 * ea * ec
                ok = (D >= 0) & (ea.abs() >= 1e-30) & (has[qx_] & has[qy_])[:, None]
                t = (-eb + pm * torch.sqrt(torch.clamp(D, min=0))) / (2 * ea)
                Tx, Ty = px * t + qx, py * t + qy
                ok = ok & (-sx * (A * Tx - C * Ty) >= 0) & (-sy * (B * Ty - C * Tx) >= 0)
                best = torch.minimum(tau[:, k], torch.where(ok, t, inf).amin((0, 1)))
                det = A * B - C * C
                dis = torch.stack([torch.sqrt(F * F * B / det)] * 2 + [torch.sqrt(F * F * A / det)] * 2)
                h = torch.stack([tx, tx, ty, ty])
                p = torch.stack([gx, gx, gy, gy]) - sa * h
                t = (pm * dis - sa * h * tn) / p
                ok = (t * tk >= tn * t0[:, kn].transpose(0, 1)) & (t > 0.5 * tn)
                ok = ok & has[:, None] & (det > 0)
                best = torch.minimum(best, torch.where(ok, t, inf).amin((0, 1)))
                tau[:, k] = torch.where(free[:, k], best, tau[:, k])
        d = (tau - old).abs() * t0
        done = (d.sum(1) / (nx * ny) < 1e-4) & (d.amax(1) < 1e-4)
        T[act[done]] = (tau * t0)[done]
        keep = ~done
        act, v = act[keep], [x[keep] for x in v]
    return T


def _adjoint(xx, yy, m, T, delta):
    """Adjoint fields [ne, n] of travel times T for the sources delta (per area)."""
    nx, ny, ne = xx.numel(), yy.numel(), T.shape[0]
    dx, dy = (xx[1] - xx[0]) * RAD, (yy[1] - yy[0]) * RAD
    co = torch.cos(yy * RAD)[:, None]
    shp = (ne, ny, nx)
    a = (m[0].reshape(-1, ny, nx) / (R * co) ** 2).expand(shp)
    b = (m[1].reshape(-1, ny, nx) / R ** 2).expand(shp)
    c = (m[2].reshape(-1, ny, nx) / (R * R * co)).expand(shp)
    t = T.reshape(shp)
    A, B = torch.zeros(shp, **F64), torch.zeros(shp, **F64)
    ty = t[:, 2:] - t[:, :-2]
    tx = t[:, :, 2:] - t[:, :, :-2]
    A[:, 1:-1, 1:] = (-(t[:, 1:-1, 1:] - t[:, 1:-1, :-1]) / dx * (a[:, 1:-1, 1:] + a[:, 1:-1, :-1]) / 2
                      + (ty[:, :, 1:] + ty[:, :, :-1]) / (4 * dy) * (c[:, 1:-1, 1:] + c[:, 1:-1, :-1]) / 2)
    B[:, 1:, 1:-1] = (-(t[:, 1:, 1:-1] - t[:, :-1, 1:-1]) / dy * (b[:, 1:, 1:-1] + b[:, :-1, 1:-1]) / 2
                      + (tx[:, 1:] + tx[:, :-1]) / (4 * dx) * (c[:, 1:, 1:-1] + c[:, :-1, 1:-1]) / 2)
    a1, a2 = A[:, 1:-1, 1:-1], A[:, 1:-1, 2:]
    b1, b2 = B[:, 1:-1, 1:-1], B[:, 2:, 1:-1]
    d = ((a2.clamp(min=0) - a1.clamp(max=0)) / dx + (b2.clamp(min=0) - b1.clamp(max=0)) / dy)
    flat = d.abs() < 1e-14
    d = torch.where(flat, 1.0, d)
    W = torch.stack([a1.clamp(min=0) / dx, -a2.clamp(max=0) / dx, b1.clamp(min=0) / dy,
                     -b2.clamp(max=0) / dy]) / d
    c0 = delta.reshape(shp)[:, 1:-1, 1:-1] / d
    W, c0 = (torch.where(flat, 0.0, v).reshape(*v.shape[:-2], -1) for v in (W, c0))
    mx, my = nx - 2, ny - 2
    ta = torch.zeros(shp, **F64)
    ta[:, 1:-1, 1:-1] = 100.0
    ta = ta.reshape(ne, -1)
    plans = []
    for xd, yd in _DIRS:
        for k in _diagonals(mx, my, xd, yd):
            plans.append((k, (k // mx + 1) * nx + k % mx + 1))
    out, act = torch.empty_like(ta), torch.arange(ne, device=DEV)
    step = torch.tensor([-1, 1, -nx, nx], device=DEV)[:, None]
    for _ in range(1000):
        old = ta.clone()
        for k, q in plans:
            ta[:, q] = c0[:, k] + (W[:, :, k] * ta[:, q + step].transpose(0, 1)).sum(0)
        ch = (ta - old).abs()
        done = (ch.sum(1) / (nx * ny) < 1e-9) & (ch.amax(1) < 1e-9)
        out[act[done]] = ta[done]
        keep = ~done
        act, ta, c0, W = act[keep], ta[keep], c0[keep], W[:, keep]
        if not act.numel():
            return out
    out[act] = ta
    return out


def _sources(xx, yy, ne, ev, lo, la, amp):
    """Point sources `amp` of events `ev` spread over cells, per km^2: [ne, n]."""
    k, w = _corners(xx * RAD, yy * RAD, lo * RAD, la * RAD)
    area = (xx[1] - xx[0]) * (yy[1] - yy[0]) * (RAD * R) ** 2 * torch.cos(la * RAD)
    d = torch.zeros((ne, xx.numel() * yy.numel()), **F64)
    return d.index_put_((ev[:, None].expand(-1, 4), k), (amp / area)[:, None] * w, accumulate=True)


def _exact_solve(c, seed):
    s = _solve_inputs(c, seed)
    xx, yy, lo, la = (_tensor(s[k]) for k in ("xx", "yy", "xrec", "yrec"))
    m = [_tensor(s[k]).reshape(1, -1) for k in ("spha", "sphb", "sphc")]
    T = _forward(xx, yy, m, _tensor(s["fun"]).reshape(1, -1), _tensor([s["x0"]]), _tensor([s["y0"]]))
    ev = torch.zeros(lo.numel(), dtype=torch.long, device=DEV)
    Ta = _adjoint(xx, yy, m, T, _sources(xx, yy, 1, ev, lo, la, _tensor(s["src"])))
    shp = (c["ny"], c["nx"])
    return dict(T=T.reshape(shp), fit=None, Ta=Ta.reshape(shp), ait=None)


def _exact_events(c, seed):
    ev, tt = _events(c, seed)
    xx, yy = (_tensor(v) for v in _grid(c))
    nx, ny = c["nx"], c["ny"]
    svel = _velocities(c, seed).reshape(c["nper"], -1)
    if c["topo"]:
        m11, m12, m22 = (m.reshape(c["nper"], -1) for m in _slopes(c, seed, c["nper"]))
    ne = ev["evlo"].size
    syn, adj, chi = [], torch.zeros_like(svel), 0.0
    part = max(1, int(4e7 / (nx * ny)))
    for e0 in range(0, ne, part):
        e = slice(e0, min(ne, e0 + part))
        ip = torch.as_tensor(ev["iper"][e], device=DEV).long()
        if c["topo"]:
            m = [m11[ip], m22[ip], -m12[ip]]
        else:
            one = torch.ones((1, nx * ny), **F64)
            m = [one, one, 0.0 * one]
        x0, y0 = _tensor(ev["evlo"][e]), _tensor(ev["evla"][e])
        T = _forward(xx, yy, m, 1.0 / svel[ip], x0, y0)
        p = slice(int(ev["rec_ptr"][e.start]), int(ev["rec_ptr"][e.stop]))
        idx = ev["rec_idx"][p]
        of = torch.as_tensor(np.repeat(np.arange(ip.numel()), np.diff(ev["rec_ptr"])[e]), device=DEV)
        lo, la = _tensor(ev["stlo"][idx]), _tensor(ev["stla"][idx])
        k, w = _corners(xx, yy, lo, la)
        t = (T[of[:, None], k] * w).sum(1)
        r = t - _tensor(tt[p])
        syn.append(t)
        chi = chi + 0.5 * (r * r).sum()
        Ta = _adjoint(xx, yy, m, T, _sources(xx, yy, ip.numel(), of, lo, la, r))
        s = c["step"]
        mx = (((xx - x0[:, None]) / s).abs() < 1.5)[:, None, :]
        my = (((yy - y0[:, None]) / s).abs() < 1.5)[:, :, None]
        Ta = torch.where((mx & my).reshape(Ta.shape), 0.0, Ta)
        adj.index_add_(0, ip, Ta * svel[ip] ** -3)
    return dict(syn=torch.cat(syn), adj_s=adj.reshape(c["nper"], ny, nx), chi=chi.reshape(1),
                fwd_iters=None, adj_iters=None, status=None)


def _exact_smooth(c, seed):
    u = _kernel(c, seed)
    ns = _nstep(c)
    ch, cv = c["sigma_h"] ** 2 / (2 * ns), c["sigma_v"] ** 2 / (2 * ns)
    h = c["step"]
    lat = torch.as_tensor(24.0 + h * np.arange(c["ny"]), **F64)[1:-1, None] * RAD
    r = 2.0 / (R - torch.as_tensor(_depths(c), **F64)[1:-1])
    fx, fy = ch / h ** 2 / torch.cos(lat) ** 2, ch * RAD * torch.tan(lat) / (2 * h)
    ix, iy, iz = (torch.arange(n, device=DEV).clamp(1, n - 2) - 1 for n in u.shape)
    for _ in range(ns):
        m = u[1:-1, 1:-1, 1:-1]
        y1, y0 = u[1:-1, 2:, 1:-1], u[1:-1, :-2, 1:-1]
        z1, z0 = u[1:-1, 1:-1, 2:], u[1:-1, 1:-1, :-2]
        d = (fx * (u[2:, 1:-1, 1:-1] + u[:-2, 1:-1, 1:-1] - 2 * m)
             + (ch / h ** 2 * (y1 + y0 - 2 * m) - fy * (y1 - y0))
             + (cv / 4.0 * (z1 + z0 - 2 * m) - cv * r / 4.0 * (z1 - z0)))
        u = (m + d)[ix][:, iy][:, :, iz]
    return [u]


def _exact_lbfgs(c, seed):
    its = _iterates(c, seed)
    s = [torch.log(b[0]) - torch.log(a[0]) for a, b in zip(its, its[1:])]
    y = [b[1] - a[1] for a, b in zip(its, its[1:])]
    rho = [1.0 / (p @ q) if p @ q > 0 else 0.0 for p, q in zip(s, y)]
    m, g = its[-1]
    q, al = g.clone(), [0.0] * len(s)
    for i in reversed(range(len(s))):
        al[i] = rho[i] * (s[i] @ q)
        q -= al[i] * y[i]
    sy, yy = s[-1] @ y[-1], y[-1] @ y[-1]
    q *= sy / yy if sy > 0 and yy > 0 else 1.0
    for i in range(len(s)):
        q += (al[i] - rho[i] * (y[i] @ q)) * s[i]
    top = q.abs().max()
    d = q / top
    angle = torch.rad2deg(torch.acos(torch.clamp(g @ d / (g.norm() * d.norm()), -1, 1)))
    vs = m * (1 - 0.02 * d)
    vp = 0.9409 + 2.0947 * vs - 0.8206 * vs ** 2 + 0.2683 * vs ** 3 - 0.0251 * vs ** 4
    ro = 1.6612 * vp - 0.4721 * vp ** 2 + 0.0671 * vp ** 3 - 0.0043 * vp ** 4 + 0.000106 * vp ** 5
    return dict(dir=d, top=float(top), angle=float(angle), model=[vs, vp, ro])


def _exact_topography(c, seed):
    s = _surface(c, seed)
    xx, yy = s["xx"], s["yy"]

    def cells(g, q):
        i = np.clip(np.searchsorted(g, q, side="right") - 1, 0, g.size - 2)
        return i, (q - g[i]) / (g[i + 1] - g[i])

    i, tx = cells(s["lon"], xx)
    j, ty = cells(s["lat"], yy)
    z, tx, ty = s["z"], tx[None, :], ty[:, None]
    j, i = j[:, None], i[None, :]
    zg = _tensor((1 - tx) * (1 - ty) * z[j, i] + tx * (1 - ty) * z[j, i + 1]
                 + (1 - tx) * ty * z[j + 1, i] + tx * ty * z[j + 1, i + 1])
    nx, ny = c["nx"], c["ny"]
    X, Y = _tensor(xx) * RAD, _tensor(yy) * RAD
    dlon = torch.sin((X[None, :] - X[:, None]) / 2) ** 2
    near = (torch.arange(nx, device=DEV)[None, :] - torch.arange(nx, device=DEV)[:, None]).abs()
    media = [[], [], [], []]
    for sig in s["sig"]:
        hx = int(3.0 * sig / (xx[1] - xx[0]))
        g = torch.empty_like(zg)
        for r in range(ny):
            c0 = math.cos(yy[r] * RAD)
            hy = int(3.0 * sig / c0 / (yy[1] - yy[0]))
            q = slice(max(0, r - hy), min(ny, r + hy + 1))
            a = (torch.sin((Y[q] - Y[r]) / 2) ** 2)[:, None, None] \
                + c0 * torch.cos(Y[q])[:, None, None] * dlon
            t = 2.0 / RAD * torch.asin(torch.sqrt(torch.clamp(a, max=1.0)))
            w = torch.exp(-t * t / (2 * sig * sig)) * (near <= hx)
            g[r] = (w * zg[q][:, None, :]).sum((0, 2)) / w.sum((0, 2))
        km = R * RAD
        dxk, dyk = (xx[1] - xx[0]) * km, (yy[1] - yy[0]) * km
        fy, fx = torch.gradient(g)
        fx, fy = fx / (dxk * torch.cos(Y)[:, None]), fy / dyk
        den = 1 + fx * fx + fy * fy
        for o, v in zip(media, ((1 + fy * fy) / den, -fx * fy / den, (1 + fx * fx) / den,
                                torch.rad2deg(torch.atan(torch.sqrt(fx * fx + fy * fy))))):
            o.append(v)
    return dict(zg=zg, media=[torch.stack(o) for o in media])


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "smooth":
        return _exact_smooth(c, seed)
    if kind == "lbfgs":
        return _exact_lbfgs(c, seed)
    if kind == "topography":
        return _exact_topography(c, seed)
    # the sweeps take one step of torch operations per anti-diagonal: grids up
    # to 420 diagonals; dispersion and eigenfunctions have no restatement here
    if kind in ("solve", "events") and c["nx"] + c["ny"] <= 420:
        return (_exact_solve if kind == "solve" else _exact_events)(c, seed)
    return None
