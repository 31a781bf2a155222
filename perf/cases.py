"""The transport path as its users call it: what a forecast, an ensemble
member, a source inversion or an output hour costs on one GPU.

A case is one restart-to-restart piece of work.  A forward case loads a
restart (FP32 ashcon and depocon held on the device, a3g_restart_load),
advances the model by a few reference time steps through the host loop a
program of its kind uses (driver.Pipeline, or driver.step where the subgrid
box has to reach the host every step), with the mass totals logged at every
step, and forms the NetCDF arrays again (a3g_output_ashcon, into device
memory).  A gradient case is one forward/adjoint pair of a source inversion.
A products case is one output hour: the 2-D products, some vertical profiles
and the NetCDF arrays of the current state.

The restart states are ash clouds some hours into an eruption: puffs along a
wind-blown track, smooth but for a few per cent of noise, heavier grains
lower down, exact zeros away from the cloud (the Crank-Nicolson solves then
give them their diffused tails, as in any run).
"""
import dataclasses
import functools
import importlib.util
import math
import pathlib
import sys

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint


def _package():
    if "volcano_ash3d_b200" not in sys.modules:
        d = pathlib.Path.cwd() / "volcano-ash3d_b200"
        spec = importlib.util.spec_from_file_location("volcano_ash3d_b200", d / "__init__.py",
                                                      submodule_search_locations=[str(d)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["volcano_ash3d_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["volcano_ash3d_b200"]


_package()
from volcano_ash3d_b200 import adjoint, driver, synthetic as syn  # noqa: E402
from volcano_ash3d_b200._lib import check  # noqa: E402
from volcano_ash3d_b200.model import Ash3dGPU  # noqa: E402

T0 = 1.2  # hours into the eruption at which a forward case restarts


def _case(name, kind, nx, ny, nz, ns, grid="projected", diffusion="cn", limiter="superbee", fast_dt=False,
          subgrid=False, terrain=False, misfit="load", slots=0, steps=2, spread=0.04):
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, ns=ns, grid=grid, diffusion=diffusion, limiter=limiter,
             fast_dt=fast_dt, subgrid=subgrid, terrain=terrain, misfit=misfit, slots=slots, steps=steps,
             spread=spread)
    return dict(c, name=name) if name else c


def listed():
    return [
        # The smallest use: one tracer bin on the 50x50x23 grid of the reference's own regression runs, explicit
        # diffusion, FAST_SUBGRID, one host call after another.  Latency and launches.
        _case("tracer 50x50x23x1", "run", 50, 50, 23, 1, diffusion="explicit", subgrid=True, steps=4, spread=0.05),
        # A local forecast (configuration C1): four grain sizes, explicit diffusion.
        _case("local 100x100x40x4", "run", 100, 100, 40, 4, diffusion="explicit", steps=6),
        # The headline step (configuration C2): quarter-degree lon/lat, ten grains, Crank-Nicolson, FAST_DT.  The
        # largest case.
        _case("regional 720x360x60x10", "run", 720, 360, 60, 10, grid="lonlat", fast_dt=True, steps=2),
        # An ensemble member (the shapes of configuration C3), odd in every extent.
        _case("member 317x211x53x7", "run", 317, 211, 53, 7, steps=4),
        # A smaller member with few grains: lines enough for part of the GPU only.
        _case("member 93x131x37x2", "run", 93, 131, 37, 2, steps=4),
        # The reference's default build, FAST_DT and FAST_SUBGRID: a cloud that fills part of its domain.
        _case("default 480x401x50x6", "run", 480, 401, 50, 6, grid="lonlat", fast_dt=True, subgrid=True, steps=4,
              spread=0.015),
        # A global one-degree run: rows that wrap around, explicit diffusion.
        _case("global 360x161x40x5", "run", 360, 161, 40, 5, grid="global", diffusion="explicit", steps=4),
        # Terrain: sigma-altitude coordinates over a mountain.
        _case("terrain 201x151x41x5", "run", 201, 151, 41, 5, terrain=True, steps=4),
        # A source inversion on hourly column loads with explicit diffusion (configuration C4), every state kept.
        _case("inversion 140x120x40x4", "gradient", 140, 120, 40, 4, diffusion="explicit"),
        # One on the deposit with Crank-Nicolson and FAST_DT (configuration C5), few checkpoints.
        _case("inversion 121x104x45x5 cn", "gradient", 121, 104, 45, 5, fast_dt=True, misfit="deposit", slots=8),
        # An output hour of a regional run.
        _case("products 480x361x50x8", "products", 480, 361, 50, 8, grid="lonlat"),
    ]


def draw(rng):
    """One more use of the same ranges: sizes spread over their logarithm, any parity."""
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    kind = rng.choice(["run"] * 7 + ["gradient", "products"])
    nx, ny, nz, ns = log(50, 500), log(50, 400), log(20, 80), log(1, 10)
    if kind == "gradient":
        nx, ny, nz, ns = log(50, 150), log(50, 130), log(20, 45), log(1, 5)
        misfit = rng.choice(["load", "deposit"])
        return _case(None, kind, nx, ny, nz, ns, diffusion=rng.choice(["cn", "explicit"]),
                     fast_dt=rng.random() < 0.5, misfit=misfit, slots=rng.choice([0, 0, 8]))
    ns = min(ns, max(1, 60_000_000 // (nx * ny * nz)))
    grid = rng.choice(["projected", "projected", "lonlat", "global"])
    if kind == "products":
        return _case(None, kind, nx, ny, nz, ns, grid=grid)
    terrain = grid == "projected" and rng.random() < 0.15
    subgrid = not terrain and rng.random() < 0.3
    return _case(None, kind, nx, ny, nz, ns, grid=grid, diffusion=rng.choice(["cn", "cn", "explicit"]),
                 limiter=rng.choice(["superbee"] * 4 + ["minmod", "mc"]), fast_dt=rng.random() < 0.5,
                 subgrid=subgrid, terrain=terrain, steps=rng.choice([2, 3, 4]),
                 spread=0.015 if subgrid else 0.04)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _config(case, seed):
    nx, ny, nz, ns = case["nx"], case["ny"], case["nz"], case["ns"]
    fall = tuple(float(v) for v in np.logspace(-3.0, math.log10(3.0), ns)) if ns > 1 else (0.1,)
    dz = 30.0 / nz if nz > 60 else max(0.5, 20.0 / nz)
    cfg = syn.Config("case", nx, ny, nz, ns, dx=5.0, dy=5.0, dz=dz, ivent=max(3, nx // 3), jvent=max(3, ny // 2),
                     fall_mps=fall, bin_mass=(1.0 / ns,) * ns, plume_km=15.0, volume_km3=1.0e-2, duration_h=3.0,
                     use_cn=case["diffusion"] == "cn", limiter=case["limiter"], sim_hours=24.0,
                     fast_subgrid=case["subgrid"], fast_dt=case["fast_dt"], seed=seed)
    if case["grid"] == "lonlat":
        cfg = dataclasses.replace(cfg, latlon=True, de=min(0.25, 350.0 / nx), dn=min(0.25, 90.0 / ny), latLL=-5.0)
    elif case["grid"] == "global":
        cfg = dataclasses.replace(cfg, latlon=True, periodic=True, de=360.0 / nx, dn=160.0 / ny, latLL=-80.0)
    if case["terrain"]:
        cfg = dataclasses.replace(cfg, zscaling_id=2, topo_km=2.0, topo_width_km=60.0)
    return cfg


@functools.lru_cache(maxsize=2)
def _geometry(key):
    return syn.geometry(_config(dict(key), 0))


def _geo(case):
    keep = ("nx", "ny", "nz", "ns", "grid", "terrain", "diffusion", "limiter", "subgrid", "fast_dt")
    return _geometry(tuple((k, case[k]) for k in keep))


def _rng(seed, stream):
    return torch.Generator(device="cuda").manual_seed(1000003 * seed + stream)


class _Met:
    """Hourly FP32 met steps: a westerly jet, a meridional wave, weak vertical motion, 5 % noise."""

    def __init__(self, cfg, seed, first, count):
        self.hours = {}
        dev = torch.device("cuda")
        x = torch.linspace(0.0, 2.0 * math.pi, cfg.nx, device=dev)
        y = torch.linspace(-1.0, 1.0, cfg.ny, device=dev)[:, None]
        z = torch.linspace(0.0, 1.0, cfg.nz, device=dev)[:, None, None]
        for h in range(first, first + count):
            g = _rng(seed, 100 + h)
            a = torch.rand(4, generator=g, device=dev)
            noise = lambda: 1.0 + 0.05 * torch.randn(cfg.nz, cfg.ny, cfg.nx, generator=g, device=dev)  # noqa: E731
            u = (4.0 + 22.0 * torch.exp(-(2.0 * y) ** 2) * torch.sin(math.pi * z)) * (0.9 + 0.2 * a[0])
            v = 6.0 * torch.sin(2.0 * x + 6.28 * a[1]) * torch.cos(0.3 * h + 2.0 * z)
            w = 0.03 * torch.sin(3.0 * x + 6.28 * a[2]) * torch.cos(2.0 * y) * torch.sin(math.pi * z)
            f = [(b * noise()).float().contiguous().cpu().numpy().transpose(2, 1, 0) for b in (u, v, w)]
            self.hours[h] = tuple(f)

    def step(self, hour):
        return self.hours[min(max(hour, min(self.hours)), max(self.hours))]


def _cloud(case, cfg, seed):
    """Restart arrays on the device: ashcon (ns, nz, ny, nx) in kg/km3 and depocon (ns, ny, nx) in kg/m2, FP32."""
    dev = torch.device("cuda")
    g = _rng(seed, 1)
    s = case["spread"]
    x = torch.arange(cfg.nx, device=dev) / cfg.nx
    y = torch.arange(cfg.ny, device=dev) / cfg.ny
    z = (torch.arange(cfg.nz, device=dev)[None, :] + 0.5) / cfg.nz
    top = min(0.8, 15.0 / (cfg.nz * cfg.dz))
    fall = torch.tensor(cfg.fall_mps, device=dev)[:, None]
    x0, y0 = cfg.ivent / cfg.nx, cfg.jvent / cfg.ny
    ash = torch.zeros(cfg.ns, cfg.nz, cfg.ny, cfg.nx, device=dev)
    dep = torch.zeros(cfg.ns, cfg.ny, cfg.nx, device=dev)
    bend = 0.6 * (torch.rand(1, generator=g, device=dev) - 0.5)
    for m in range(5):
        r = torch.rand(3, generator=g, device=dev)
        wide = s * (0.6 + 0.25 * m) * (0.8 + 0.4 * r[0])
        ex = torch.exp(-0.5 * ((x - x0 - 1.6 * s * m) / wide) ** 2)
        ey = torch.exp(-0.5 * ((y - y0 - 1.6 * s * m * bend - s * (r[1] - 0.5)) / wide) ** 2)
        h = (top * (0.9 - 0.1 * m) / (1.0 + 0.3 * fall * m)).clamp(min=0.02)
        ez = torch.exp(-0.5 * ((z - h) / 0.08) ** 2)
        pz = 1.0e5 / (1.0 + m) * (0.5 + r[2]) * ez
        ash += pz[:, :, None, None] * (ey[:, None] * ex[None, :])
        dep += (1.0e-2 * fall)[:, :, None] * (ey[:, None] * ex[None, :])
    for q in range(cfg.ns):
        ash[q] *= 1.0 + 0.03 * torch.randn(ash[q].shape, generator=g, device=dev).clamp(-3.0, 3.0)
    ash[ash < 1.0e-9] = 0.0
    dep[dep < 1.0e-6] = 0.0
    return ash, dep


def _observations(case, cfg, seed):
    """What an inversion is given: hourly column loads (nx, ny) or a deposit thickness (nx, ny), and a first guess
    of the source, (nz, hours, ns) in kg/h."""
    g = np.random.default_rng(seed)
    x = (np.arange(cfg.nx) - cfg.ivent)[:, None] / cfg.nx
    y = (np.arange(cfg.ny) - cfg.jvent)[None, :] / cfg.ny
    blob = np.exp(-((x - 0.1) / 0.15) ** 2 - (y / 0.1) ** 2) * (1.0 + 0.05 * g.standard_normal((cfg.nx, cfg.ny)))
    col = syn.suzuki_column(cfg)[:cfg.nz]
    rate = syn.mass_flux_rate(cfg) * col[:, None, None] * np.asarray(cfg.bin_mass)[None, None, :]
    return 10.0 * blob, 0.1 * blob, np.ascontiguousarray(rate * np.exp(0.5 * g.standard_normal((cfg.nz, 1, cfg.ns))))


# ---------------------------------------------------------------------------
# the work
# ---------------------------------------------------------------------------
def prepare(case, seed):
    cfg = _config(case, seed)
    model = Ash3dGPU(cfg, geo=_geo(case))
    s = dict(case=case, cfg=cfg, model=model)
    if case["kind"] == "gradient":
        load, dep, s["p"] = _observations(case, cfg, seed)
        by_load = case["misfit"] == "load"
        level = 8.0 * ((cfg.nx + 7) // 8 * 8) * cfg.ny * cfg.nz * cfg.ns
        s["inv"] = adjoint.InversionGPU(model, cfg, 1, obs={0: load} if by_load else None,
                                        obs_dep=None if by_load else dep, fast_dt=cfg.fast_dt,
                                        snapshot_bytes=(case["slots"] + 0.5) * level if case["slots"] else 0.0,
                                        met=_Met(cfg, seed, 0, 3))
        return s
    s["ash"], s["dep"] = _cloud(case, cfg, seed)
    s["out"], s["out_dep"] = torch.empty_like(s["ash"]), torch.empty_like(s["dep"])
    torch.cuda.synchronize()
    if case["kind"] == "products":
        check(model.lib.a3g_restart_load(model.ctx, s["ash"].data_ptr(), s["dep"].data_ptr()))
        model.set_output_params()
        model.output_reset()
        s["points"] = [(cfg.ivent + d, cfg.jvent) for d in range(0, cfg.nx - cfg.ivent, max(1, cfg.nx // 12))]
        return s
    hour = int(T0)
    met = _Met(cfg, seed, hour, 2)
    model.set_met_steps(met.step(hour), met.step(hour + 1))
    if cfg.fast_subgrid:
        st = driver.new_state(cfg, model.geo)
    else:
        s["loop"] = driver.Pipeline(model, cfg, model.geo)
        st = s["loop"].st
    st.met, st.hour, st.met_ahead, st.time = met, hour, hour + 2, T0
    if cfg.fast_dt:
        driver.meso_dt(model, st, "pair", cfg.sim_hours, cfg.sim_hours)
    model.sync()
    s["start"] = st
    return s


def run(s):
    case, model = s["case"], s["model"]
    if case["kind"] == "gradient":
        J, loads, dep = s["inv"].forward(s["p"])
        return dict(J=J, loads=loads, dep=dep, grad=s["inv"].adjoint())
    if case["kind"] == "products":
        products = model.output_vars(T0)
        profiles, written = model.vprofiles(s["points"])
        check(model.lib.a3g_output_ashcon(model.ctx, s["out"].data_ptr(), s["out_dep"].data_ptr()))
        return dict(products, profiles=profiles, written=written, ashcon=s["out"], depocon=s["out_dep"])
    check(model.lib.a3g_restart_load(model.ctx, s["ash"].data_ptr(), s["dep"].data_ptr()))
    st = dataclasses.replace(s["start"], history=[])
    if "loop" in s:
        loop = s["loop"]
        loop.st, loop.state = st, [1, 1]
        for _ in range(case["steps"]):
            loop.step()
        loop.flush()
    else:
        for _ in range(case["steps"]):
            driver.step(model, st)
    check(model.lib.a3g_output_ashcon(model.ctx, s["out"].data_ptr(), s["out_dep"].data_ptr()))
    # the outflow accumulators go on from pass to pass (a restart does not reset them), so their total is no
    # function of the inputs; everything else of the log is
    log = np.array([(r.dt, r.time, r.aloft, r.dep, r.source_cum) for r in st.history])
    return dict(ashcon=s["out"], depocon=s["out_dep"], log=log)


def work(case):
    """Bytes: the state read and written once per step and the met steps it is moved by, the FP32 restart arrays
    in and out; operations: the reference's per cell and grain (about 40 an advection sweep, 14 a Crank-Nicolson
    and 8 an explicit diffusion sweep).  A subgrid run cannot do without reading the state to find its box, and
    moves the cloud's share of it."""
    cells = case["nx"] * case["ny"] * case["nz"]
    cg = cells * case["ns"]
    sweep = 3 * 40 + 3 * (14 if case["diffusion"] == "cn" else 8)
    if case["kind"] == "products":
        return dict(bytes=8 * cg + 4 * cg + 80 * case["nx"] * case["ny"], flops=3 * cg)
    if case["kind"] == "gradient":  # one hour of about 25 steps, each run forward, stored, and reversed
        return dict(bytes=25 * cg * (16 + 8 + 8 + 16) + 25 * 48 * cells, flops=25 * 3 * sweep * cg)
    if case["subgrid"]:
        share = min(1.0, 32.0 * case["spread"]) * min(1.0, 24.0 * case["spread"]) * 0.9
        return dict(bytes=case["steps"] * (8 * cg + 16 * share * cg + 24 * cells) + 8 * cg,
                    flops=case["steps"] * sweep * share * cg)
    return dict(bytes=case["steps"] * (16 * cg + 24 * cells) + 8 * cg, flops=case["steps"] * sweep * cg)


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------
class _Plain:
    """The reference's step on (ns, nz, ny, nx) tensors.  Axis d of a sweep: 3 (x), 2 (y), 1 (z).  Geometry and
    winds carry two ghost cells at either end of every axis, (1, nz+4, ny+4, nx+4)."""

    EPS, DT_MIN, DT_MAX = 1.0e-10, 1.0e-5, 1.0

    def __init__(self, case, cfg, geo):
        self.case, self.cfg, self.dev = case, cfg, torch.device("cuda")
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a.T), device=self.dev)[None]  # noqa: E731
        self.kap = t(geo["kappa"])
        self.sig = {3: t(geo["sig_nx"]), 2: t(geo["sig_ny"]), 1: t(geo["sig_nz"])}
        self.dz = torch.as_tensor(geo["dz_vec"], device=self.dev)
        self.fall = torch.tensor([-v * 3.6 for v in cfg.fall_mps], dtype=torch.float64, device=self.dev)
        self.k = cfg.diffusivity_m2s * 3.6e-3
        self.n = {3: cfg.nx, 2: cfg.ny, 1: cfg.nz}
        self.box = {d: (1, self.n[d]) for d in self.n}
        self.limit = None
        if case["terrain"]:
            f = syn.topo_fields(cfg)
            self.slope = [t(f["dhdx"][..., None])[:, :, 2:-2, 2:-2], t(f["dhdy"][..., None])[:, :, 2:-2, 2:-2]]
            self.deld = {3: t(f["deldx"][..., None]), 2: t(f["deldy"][..., None])}
            self.level = torch.as_tensor(f["s_cc"][2:-2] / f["ztop"] - 1.0, device=self.dev)[None, :, None, None]

    def inner(self, a, but=None):
        """The interior of a ghosted array, axis `but` left ghosted."""
        for d in (1, 2, 3):
            if d != but and a.shape[d] > 1:
                a = a.narrow(d, 2, a.shape[d] - 4)
        return a

    def winds(self, last, nxt, frac):
        self.met = [[torch.as_tensor(np.ascontiguousarray(a.T), device=self.dev)[None] for a in m] for m in (last, nxt)]
        self.v = [(a.double() + (b - a).double() * frac) * 3.6 for a, b in zip(*self.met)]
        self.vz_ghost = self.v[2]
        if self.case["terrain"]:
            self.v[2] = self.v[2] + self.level * (self.v[0] * self.slope[0] + self.v[1] * self.slope[1])

    # --- dt -----------------------------------------------------------------
    def limits(self):
        if self.limit is None:
            total = 0.0
            for d in (3, 2, 1):
                s = self.inner(self.sig[d], d)
                m = torch.minimum(s.narrow(d, 2, self.n[d]), s.narrow(d, 3, self.n[d]))
                total = total + (self.inner(self.kap) / m) ** 2 / self.k
            t = min(self.DT_MAX, float(total.min()))
            self.limit = t * 4.0 if self.cfg.use_cn else t * 0.5
        return self.limit

    def courant(self, v, fall):
        dx, dy = syn.projected_dxdy(self.cfg)
        m = []
        for d, a, h in ((3, v[0], dx), (2, v[1], dy)):
            if self.cfg.latlon:
                s = self.inner(self.sig[d], d)
                a = a.abs() * torch.minimum(s.narrow(d, 2, self.n[d]), s.narrow(d, 3, self.n[d])) / self.inner(self.kap)
                m.append(float(a.max()))
            else:
                m.append(float(a.abs().max()) / h)
        m.append(float((fall / self.dz[2:-2][None, :, None, None]).max()))
        dt = min(1.0 / max(m), self.limits())
        dt = self.DT_MIN if dt < self.DT_MIN else self.DT_MAX if dt > self.DT_MAX else self.cfg.cfl * dt
        return self.DT_MIN * int(dt / self.DT_MIN)

    def clip(self, dt, time, write, end):
        if 1.0e-6 < write - time < dt:
            dt = write - time
        return end - time if time + dt > end else dt

    def adjust_dt(self, time, write, end):
        return self.clip(self.courant(self.v, self.vz_ghost.abs() + self.fall.abs().max()), time, write, end)

    def meso_dt(self, m, time, write, end):
        vf = torch.tensor([-1.0 * f for f in self.cfg.fall_mps], dtype=torch.float32, device=self.dev).abs().max()
        return self.clip(self.courant([m[0].double().abs() * 3.6, m[1].double().abs() * 3.6],
                                      (m[2].abs() + vf).double() * 3.6), time, write, end)

    # --- sweeps -------------------------------------------------------------
    def in_box(self, q, but=None):
        m = torch.ones((), dtype=torch.bool, device=self.dev)
        for d in (1, 2, 3):
            if d != but:
                i = torch.arange(1, self.n[d] + 1, device=self.dev)
                shape = [1, 1, 1, 1]
                shape[d] = -1
                m = m & ((i >= self.box[d][0]) & (i <= self.box[d][1])).view(shape)
        return m

    def ghosted(self, a, d, how):
        if how == "wrap":
            return torch.cat([a.narrow(d, self.n[d] - 2, 2), a, a.narrow(d, 0, 2)], d)
        lo, hi = a.narrow(d, 0, 1), a.narrow(d, self.n[d] - 1, 1)
        if how == "zero":
            lo, hi = torch.zeros_like(lo), torch.zeros_like(hi)
        return torch.cat([lo, lo, a, hi, hi], d)

    def advect(self, q, d, dt):
        """The sweep along axis d; gives the state and, for z, what left through the ground."""
        n, (lo, hi) = self.n[d], self.box[d]
        wrap = self.cfg.periodic and d == 3
        at = torch.arange(-1, n + 3, device=self.dev)
        shape = [1, 1, 1, 1]
        shape[d] = n + 4
        at = at.view(shape)
        qe = self.ghosted(q, d, "wrap" if wrap else "zero")
        qe = torch.where((at >= lo - 2) & (at <= hi + 2), qe, 0.0)
        ve = self.ghosted(self.v[3 - d], d, "wrap" if wrap else "edge")
        if d == 1:
            g = self.ghosted(self.vz_ghost, d, "edge")
            ve = torch.where((at < 1) | (at > n), g, ve) + self.fall[:, None, None, None]
        sig, dtv = self.inner(self.sig[d], d), dt / self.inner(self.kap, d)
        back = lambda a: torch.cat([torch.zeros_like(a.narrow(d, 0, 1)), a.narrow(d, 0, n + 3)], d)  # noqa: E731
        ahead = lambda a: torch.cat([a.narrow(d, 1, n + 3), torch.zeros_like(a.narrow(d, 0, 1))], d)  # noqa: E731
        fs_ok, fss_ok = (at >= lo - 1) & (at <= hi + 1), (at >= lo) & (at <= hi + 1)
        us = torch.where(fs_ok, 0.5 * (back(ve) + ve) * sig, 0.0)
        dq = qe - back(qe)
        dqu = torch.where(us > 0.0, back(dq), ahead(dq))
        pos, neg = us.clamp(min=0.0), us.clamp(max=0.0)
        skip = (dq.abs() <= self.EPS) | ~fss_ok
        big = dqu.abs() > 3.0 * dq.abs()
        theta = torch.where(big, torch.copysign(torch.full_like(dq, 3.0), dqu * dq),
                            torch.where(skip | big, 1.0, dqu) / torch.where(skip, 1.0, dq))
        fss = torch.where(skip, 0.0, 0.5 * us.abs() * (1.0 - dtv * us.abs()) * (dq * self.limiter(theta)))
        fr = pos * dq + qe * (ahead(neg) - neg)
        fl = neg * dq + back(qe) * (pos - back(pos))
        if self.case["terrain"] and d != 1:
            deld = self.deld[d].narrow(5 - d, 2, self.n[5 - d]) if d == 3 else self.deld[d].narrow(3, 2, self.n[3])
            tt = 0.5 * ve * (sig + ahead(sig)) * qe * torch.where(fs_ok, deld, 0.0)
            fr, fl = fr + tt, fl - back(tt)
        fr, fl = torch.where(fs_ok, fr, 0.0), torch.where(fs_ok, fl, 0.0)
        upd = -(dtv * (ahead(fl) + fr + ahead(fss) - fss))
        new = torch.where((at >= lo) & (at <= hi), qe + upd, 0.0).narrow(d, 2, n)
        new = torch.where(self.in_box(q, d), new, 0.0)
        ground = None
        if d == 1 and lo == 1:
            ground = torch.where(self.in_box(q, 1)[:, 0], upd[:, 1], 0.0)
        return new, ground

    def limiter(self, t):
        if self.cfg.limiter == "minmod":
            return torch.where(t > 1.0, 1.0, torch.where(t > 0.0, t, 0.0))
        if self.cfg.limiter == "mc":
            m = torch.where((1.0 + t) / 2.0 < 2.0, (1.0 + t) / 2.0, 2.0)
            m = torch.where(m < 2.0 * t, m, 2.0 * t)
            return torch.where(m > 0.0, m, 0.0)
        return torch.where(t > 2.0, 2.0, torch.where(t > 1.0, t, torch.where(t > 0.5, 1.0, torch.where(t > 0.0, 2.0 * t, 0.0))))

    def weights(self, d, dt):
        """dt*k_ds*sigma/kappa of either face of every cell of axis d, ghosts of the sweep axis off."""
        n = self.n[d]
        s, kp = self.inner(self.sig[d], d), self.inner(self.kap, d)
        c = lambda a, o: a.narrow(d, 2 + o, n)  # noqa: E731
        left = dt * self.k * (c(s, 0) / (0.5 * (c(kp, -1) + c(kp, 0)))) * c(s, 0) / c(kp, 0)
        right = dt * self.k * (c(s, 1) / (0.5 * (c(kp, 0) + c(kp, 1)))) * c(s, 1) / c(kp, 0)
        return left, right

    def diffuse(self, q, d, dt):
        n, (lo, hi) = self.n[d], self.box[d]
        left, right = self.weights(d, dt)
        if not self.cfg.use_cn:
            e = self.ghosted(q, d, "wrap" if self.cfg.periodic and d == 3 else "edge")
            new = q + (right * (e.narrow(d, 3, n) - q) - left * (q - e.narrow(d, 1, n)))
            return torch.where(self.in_box(q), new, 0.0)
        if hi == lo:
            return q
        row = lambda a: a.narrow(d, lo - 1, hi - lo + 1).movedim(d, 0)  # noqa: E731
        x, L, R, m = row(q), row(left), row(right), hi - lo + 1
        xm = torch.cat([x[:1], x[:-1]])
        xp = torch.cat([x[1:], x[-1:]])
        b = 0.5 * L * xm + (1.0 - 0.5 * (L + R)) * x + 0.5 * R * xp
        diag = 1.0 + 0.5 * (L + R)
        diag = torch.cat([diag[:1] - 0.5 * L[:1], diag[1:-1], diag[-1:] - 0.5 * R[-1:]])
        p, y = [diag[0]], [b[0]]
        for i in range(1, m):
            f = -(0.5 * L[i]) / p[-1]
            p.append(diag[i] + f * (0.5 * R[i - 1]))
            y.append(b[i] - f * y[-1])
        out = [y[-1] / p[-1]]
        for i in range(m - 2, -1, -1):
            out.append((y[i] + 0.5 * R[i] * out[-1]) / p[i])
        new = torch.stack(out[::-1]).movedim(0, d)
        size = list(new.shape)
        size[d] = lo - 1
        before = new.new_zeros(size)
        size[d] = n - hi
        return torch.where(self.in_box(q), torch.cat([before, new, new.new_zeros(size)], d), 0.0)

    def find_box(self, q):
        """get_minmax_index, the vent at (ivent, jvent, 1)."""
        vent = {3: self.cfg.ivent, 2: self.cfg.jvent, 1: 1}
        hot = q.amax(0) >= 1.0e-7
        for d in (3, 2, 1):
            n = self.n[d]
            f = hot.movedim(d - 1, 0).reshape(n, -1).any(1).tolist()
            a, b = 1, n
            for i in range(2, vent[d]):
                if f[i - 1]:
                    break
                a = i
            for i in range(n, a + 1, -1):
                if f[i - 1]:
                    break
                b = i
            if d == 3 and self.cfg.periodic and (a == 1 or b == n):
                a, b = 1, n
            if b - a < 2:
                b = min(b + 1, n)
                a = b - 2
            self.box[d] = (a, b)

    def step(self, q, itime, dt):
        """Set_BC ... DiffuseVert of one step."""
        if self.cfg.fast_subgrid:
            self.find_box(q)
        for d in ((2, 3) if itime % 2 == 0 else (3, 2)):
            q, _ = self.advect(q, d, dt)
        q, ground = self.advect(q, 1, dt)
        if self.cfg.fast_subgrid:
            self.box = {d: (max(1, a - 1), min(self.n[d], b + 1)) for d, (a, b) in self.box.items()}
        for d in ((3, 2) if itime % 2 == 0 else (2, 3)):
            q = self.diffuse(q, d, dt)
        return self.diffuse(q, 1, dt), ground


def exact(case, seed):
    cfg = _config(case, seed)
    one = _Plain(case, cfg, _geo(case))
    if case["kind"] == "gradient":
        return _exact_gradient(case, cfg, one, seed)
    ash, depo = _cloud(case, cfg, seed)
    if case["kind"] == "products":
        return _exact_products(case, cfg, one, ash, depo)
    q, ground = ash.double(), depo.double()
    hour = int(T0)
    met = _Met(cfg, seed, hour, 2)
    pair = met.step(hour), met.step(hour + 1)
    col = torch.as_tensor(syn.suzuki_column(cfg)[:cfg.nz], device=one.dev)
    rate = torch.tensor(cfg.bin_mass, dtype=torch.float64, device=one.dev)[:, None] * syn.mass_flux_rate(cfg) * col
    kcol = one.inner(one.kap)[0, :, min(cfg.jvent - 1, one.inner(one.kap).shape[2] - 1), cfg.ivent - 1]
    time, poured, log = T0, 0.0, []
    for itime in range(1, case["steps"] + 1):
        one.winds(*pair, time - hour)
        if cfg.fast_dt:
            a, b = (one.meso_dt(m, T0, cfg.sim_hours, cfg.sim_hours) for m in one.met)
            dt = one.clip(a + (b - a) * (time - hour), time, cfg.sim_hours, cfg.sim_hours)
        else:
            dt = one.adjust_dt(time, cfg.sim_hours, cfg.sim_hours)
        share = (min(time + dt, cfg.duration_h) - time) / dt
        q[:, :, cfg.jvent - 1, cfg.ivent - 1] += dt * share * rate / kcol
        poured += float((dt * share * rate).sum()) / cfg.magma_density / 1.0e9
        q, fell = one.step(q, itime, dt)
        if fell is not None:
            ground = ground + fell
        time += dt
        aloft = float((q * one.inner(one.kap)).sum()) / cfg.magma_density / 1.0e9
        down = float((ground * one.inner(one.kap, 1)[:, 1]).sum()) / cfg.magma_density / 1.0e9
        log.append((dt, time, aloft, down, poured))
    return dict(ashcon=q, depocon=_depocon(one, ground), log=np.array(log))


def _depocon(one, ground):
    d = ground * one.dz[1] / 1.0e6
    return torch.where(d.float().double() <= 1.0e-6, 0.0, d)


def _exact_products(case, cfg, one, ash, depo):
    c, ground = ash.double(), depo.double()
    f = lambda a: np.asfortranarray(a.cpu().numpy().T)  # noqa: E731
    total = c[0].clone()
    for g in range(1, cfg.ns):
        total = total + c[g]
    zcc = torch.as_tensor(syn.zgrid(cfg)[1][2:-2], device=one.dev)[:, None, None]
    dz = one.dz[2:-2][:, None, None]
    load = torch.zeros_like(total[0])
    for k in range(cfg.nz):
        load = load + total[k] * dz[k] / 1.0e3
    thick = ground.sum(0) * one.dz[2] / 1.0e6 / 1000.0 * 1.0e3
    seen, covered = load >= 0.2, thick > 1.0e-2
    top = torch.where(total >= 1.0e-3, zcc + 0.5 * dz, 0.0).amax(0)
    base = torch.where(total <= 1.0e-3, zcc - 0.5 * dz, 100.0).amin(0)
    base = torch.minimum(top, torch.where((base < 0.0) & (top > 0.0), 0.0, base))
    mask = lambda a: torch.where(seen, a, 0.0)  # noqa: E731
    area = one.inner(one.sig[1])[0, 0].expand(cfg.ny, cfg.nx)
    points = [(cfg.ivent + d, cfg.jvent) for d in range(0, cfg.nx - cfg.ivent, max(1, cfg.nx // 12))]
    heavy = [bool(c[:, :, j - 1, i - 1].sum() >= 1.0e-3) for i, j in points]
    prof = np.stack([total[:, j - 1, i - 1].cpu().numpy() * 1.0e-3 for i, j in points], 1)
    hours = lambda h: torch.full_like(load, h)  # noqa: E731
    late = lambda m: f(torch.where(m, hours(T0), hours(-1.0)))  # noqa: E731
    return dict(cloud_load=f(mask(load)), max_height=f(mask(top)), min_height=f(mask(base)),
                max_conc=f(mask(total.amax(0) * 1.0e-3)), dep_thick=f(thick), cloud_arrival=late(seen),
                dep_arrival=late(covered), mask_cloud=f(seen), mask_dep=f(covered),
                cloud_area=float(area[seen].sum()), dep_area=float(area[covered].sum()), cloud_load_area=None,
                profiles=prof, written=np.array(heavy, dtype=np.int32), ashcon=c, depocon=_depocon(one, ground))


def _exact_gradient(case, cfg, one, seed):
    """The misfit, its observations, and its gradient by torch's reverse mode, a step recomputed at a time."""
    load_obs, dep_obs, p = _observations(case, cfg, seed)
    met = _Met(cfg, seed, 0, 3)
    p = torch.as_tensor(p, device=one.dev).requires_grad_()
    kcol = one.inner(one.kap)[0, :, cfg.jvent - 1, cfg.ivent - 1]
    q = torch.zeros(cfg.ns, cfg.nz, cfg.ny, cfg.nx, dtype=torch.float64, device=one.dev)
    ground = torch.zeros_like(q[:, 0])
    time, itime = 0.0, 0
    one.winds(met.step(0), met.step(1), 0.0)
    if cfg.fast_dt:
        a, b = (one.meso_dt(m, 0.0, 1.0, 1.0) for m in one.met)

    def advance(q, p, winds, itime, dt):
        one.v, one.vz_ghost = winds
        at = torch.zeros(cfg.ny, cfg.nx, dtype=torch.float64, device=one.dev)
        at[cfg.jvent - 1, cfg.ivent - 1] = 1.0
        q = q + dt * (p[:, 0].T / kcol)[:, :, None, None] * at
        return one.step(q, itime, dt)

    while time < 1.0 - 1.0e-12:
        itime += 1
        one.winds(met.step(0), met.step(1), time)
        dt = one.clip(a + (b - a) * time, time, 1.0, 1.0) if cfg.fast_dt else one.adjust_dt(time, 1.0, 1.0)
        q, fell = checkpoint(advance, q, p, (one.v, one.vz_ghost), itime, dt, use_reentrant=False)
        ground = ground + fell
        time += dt
    load = (q.sum(0) * one.dz[2:-2][:, None, None] / 1.0e3).sum(0)
    thick = ground.sum(0) * one.dz[2] / 1.0e6 / 1000.0 * 1.0e3
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a.T), device=one.dev)  # noqa: E731
    miss = load - t(load_obs) if case["misfit"] == "load" else thick - t(dep_obs)
    J = 0.5 * (miss * miss).sum()
    J.backward()
    f = lambda a: a.detach().cpu().numpy()  # noqa: E731
    return dict(J=float(J.detach()), loads=np.ascontiguousarray(f(load).T)[None], dep=np.ascontiguousarray(f(thick).T),
                grad=f(p.grad))
