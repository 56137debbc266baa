"""The work that users of this framework have it do, as cases to be timed.

A case is one of six kinds of use, each through the public entry points:

stage     one explicit RK stage of one tracer on device arrays that the
          caller owns (``olamgpu_update_scalar_noalloc``): the call of a
          program that must not allocate
steps     tracer steps under given winds, state resident on the device
          (``scalar_transport_rk``): off-line transport
limited   the same with the monotonic (1) or the positive-definite (2)
          limiter
long      long steps of the whole dynamical core, recorded as a CUDA graph
          (``timestep``): acoustic RK3 steps with damping, the tracer step
window    a window of long steps with checkpoints and a surface emission,
          and the adjoint of its transport (``window_forward`` and
          ``window_adjoint``): one iteration of an inversion
dropin    one tracer step in the literal drop-in mode: every call uploads
          its inputs from the host arrays and downloads its outputs

In the resident kinds a pass writes a new state into the host arrays that
the library was given (from the GPU, where the state was made), sends them
to the device, runs the steps and fetches the results: what a host model
does around a block of device steps.  Sizes are those of the repository's
benchmark configurations (NXP = 20, 100, 200 divisions of the icosahedron,
30 and 60 levels, 1, 5, 32 and 128 tracers) and odd ones between them.

``exact`` restates the path in 64 bits with plain torch operations.
"""
import ctypes
import functools
import math

import numpy as np
import torch

from olam_b200 import abi
from olam_b200.lib import HostState, OlamGpu, check
from olam_b200.synth.grid import build_grid, stretched_levels, with_terrain

R_DRY, CP, CV, GRAV, P00, ERAD = 287.0, 1004.0, 717.0, 9.81, 1.0e5, 6371.22e3
ALPHA = np.float32((1.0 / P00) ** (R_DRY / CV) * R_DRY ** (CP / CV))
NACOUST = 4          # acoustic steps per long step
EXACT_TRACERS = 8    # the exact tracers of a case with more of them than that


def _case(name, kind, nxp, nlev, ntr, steps, order=2, nrk=2, monot=0, terrain=0):
    c = dict(kind=kind, nxp=nxp, nlev=nlev, ntr=ntr, steps=steps, order=order, nrk=nrk, monot=monot,
             terrain=terrain)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: one tracer, one stage, the 4002-column grid
        _case("stage nxp20", "stage", 20, 30, 1, 1),
        # the largest grid that the call takes at third order
        _case("stage nxp58 order3", "stage", 58, 60, 1, 1, order=3),
        # one passive tracer on the small configuration, ten RK3 steps of 300 s
        _case("steps nxp20 x1", "steps", 20, 30, 1, 10, nrk=3),
        # an odd chemistry set over mountains at third order
        _case("steps nxp47 x33 terrain", "steps", 47, 41, 33, 24, order=3, nrk=3, terrain=4),
        # the batched headline: 128 tracers, 60 levels (a quarter of its columns)
        _case("steps nxp100 x128", "steps", 100, 60, 128, 48),
        # aerosol and moisture species that must stay positive
        _case("positive nxp60 x16", "limited", 60, 60, 16, 12, monot=2),
        # monotonic transport at third order, odd sizes
        _case("monotonic nxp37 x9", "limited", 37, 43, 9, 12, order=3, nrk=3, monot=1),
        # the whole core on the small configuration: launches and latency
        _case("long nxp20 x1", "long", 20, 30, 1, 10, nrk=3),
        # the whole core, 5 tracers (the full dynamics configuration)
        _case("long nxp100 x5", "long", 100, 60, 5, 8),
        # the whole core on the largest grid whose state fits three times
        _case("long nxp200 x16", "long", 200, 60, 16, 6),
        # an inversion's iteration: 32 tracers, 12 steps, checkpoints every 4
        _case("window nxp64 x32", "window", 64, 60, 32, 12, nrk=3),
        # one call as OLAM's Fortran makes it, host arrays in and out
        _case("dropin nxp60 x24", "dropin", 60, 60, 24, 1),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["stage", "steps", "steps", "limited", "long", "long", "window", "dropin"])
    order, nrk, nlev = rng.choice([2, 2, 3]), rng.choice([2, 3]), log(12, 80)
    if kind == "stage":
        return _case(None, kind, log(8, 50), nlev, 1, 1, order)
    if kind == "dropin":
        return _case(None, kind, log(10, 60), nlev, log(1, 40), 1, order, nrk)
    if kind == "window":
        return _case(None, kind, log(10, 50), nlev, log(2, 32), 4 * rng.randint(1, 3), 2, nrk)
    nxp = log(8, 90)
    # tracers of all steps together within the listed cases' columns and levels
    most = max(1, min(128, int(7.0e8 / (10.0 * nxp * nxp * nlev * 12))))
    if kind == "limited":
        return _case(None, kind, nxp, nlev, log(1, min(most, 32)), rng.randint(6, 12), order, nrk, rng.choice([1, 2]))
    if kind == "long":
        return _case(None, kind, nxp, nlev, log(1, min(most, 32)), rng.randint(4, 8), 2, nrk)
    return _case(None, kind, nxp, nlev, log(1, most), rng.randint(10, 40), order, nrk, terrain=rng.choice([0, 0, 4]))


def _dt(case):
    """Long step [s]: 300 s at NXP = 20, 120 s at 100, 60 s at 200."""
    return min(300.0, 12000.0 / case["nxp"])


def _dynamic(case):
    return case["kind"] in ("long", "window")


# ---- grid and model handle ---------------------------------------------------

@functools.lru_cache(maxsize=1)
def _grid(nxp, nlev, terrain):
    g = build_grid(nxp, stretched_levels(nlev, 100.0, 30000.0), seed=5)
    return with_terrain(g, terrain) if terrain else g


def _grid_of(case):
    return _grid(case["nxp"], case["nlev"], case["terrain"])


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


@functools.lru_cache(maxsize=1)
def _tables(nxp, nlev, terrain):
    """The grid's tables as torch tensors: indices, masks, 64-bit metrics."""
    g, dev = _grid(nxp, nlev, terrain), _device()
    t = {}
    for k in ("itab_w_iw", "itab_w_iv", "itab_v_iw", "itab_v_im", "itab_m_iv", "itab_m_im"):
        t[k] = torch.from_numpy(np.ascontiguousarray(getattr(g, k)).astype(np.int64)).to(dev)
    for k in ("gxps_coef", "gyps_coef", "xy_h", "xy_hu", "dxps", "dyps", "xx0_v", "xy0_v", "yy0_v", "xx0_vu",
              "xy0_vu", "yy0_vu", "a_w", "a_wu", "volti", "volt", "arv", "arw", "volwi", "volvi", "arw0", "arm0",
              "dniv", "dniu", "dnv", "zfacit", "dzit", "zt", "zm", "xx_yy", "xx_yy_m", "wnx", "wny", "wnz", "wnxo2",
              "wnyo2", "wnzo2", "vnx", "vny", "vnz", "ecvec_vx", "ecvec_vy", "ecvec_vz", "gdz_wgtm", "gdz_wgtp",
              "gdz_wgtm8", "gdz_wgtp8", "zwgt_top8", "zwgt_bot8", "dzim", "glatw", "glonw", "glatv", "glonv"):
        t[k] = torch.from_numpy(np.array(getattr(g, k), dtype=np.float64)).to(dev)
    poly = torch.from_numpy(np.asarray(g.npoly).astype(np.int64)).to(dev)
    t["valid"] = torch.arange(7, device=dev)[None] < poly[:, None]
    t["dirv"] = torch.from_numpy(np.array(g.dirv, np.float64)).to(dev) * t["valid"]
    lev = torch.arange(g.mza, device=dev)[None]
    t["kw"] = torch.from_numpy(np.asarray(g.lpw).astype(np.int64) - 1).to(dev)     # lowest level of a column
    t["open_w"] = lev >= t["kw"][:, None]
    t["open_v"] = lev >= torch.from_numpy(np.asarray(g.lpv).astype(np.int64) - 1).to(dev)[:, None]
    return t


def _tables_of(case):
    return _tables(case["nxp"], case["nlev"], case["terrain"])


class _Model:
    """The library's handle (one per process) with the host arrays it was
    given, as a host model keeps them for its whole run."""

    def __init__(self, case):
        g = self.grid = _grid_of(case)
        self.fgrid = abi.FortranGrid(g)
        kind, n = case["kind"], case["ntr"]
        self.opts = abi.make_opts(_dt(case), nacoust=NACOUST, nrk_scal=case["nrk"], scal_order=case["order"],
                                  iscal_monot=case["monot"])
        w, v = (g.mwa, g.mza), (g.mva, g.mza)

        def pinned(shape, dtype=torch.float32):
            return torch.zeros(shape, dtype=dtype, pin_memory=True)

        arrays = dict(rho=pinned(w, torch.float64), vmasc=pinned(v), wmasc=pinned(w), wc=pinned(w))
        if _dynamic(case):
            arrays |= {k: pinned(w) for k in ("thil", "wmc", "vxe", "vye", "vze")}
            arrays |= {k: pinned(v) for k in ("vmc", "vc")}
            arrays["press"] = pinned(w, torch.float64)
            constant = dict(alpha_press=np.full(w, ALPHA, np.float32),
                            pwfac=np.broadcast_to(g.dzim, w).astype(np.float32),
                            pvfac=(g.zfacit[None] * g.dniv[:, None]).astype(np.float32), vmt=np.zeros(v, np.float32))
            constant |= {k: np.zeros(w, np.float32) for k in ("thilt", "vmxet", "vmyet", "vmzet")}
        else:
            constant = {}
        self.arrays = arrays
        self.host = HostState(**{k: a.numpy() for k, a in arrays.items()}, **constant)
        self.dev = OlamGpu(self.fgrid, self.opts, self.host)
        self.rho_old = pinned(w)
        if kind != "stage":
            self.tracers, self.tend = pinned((n, *w)), pinned((n, *w))
            self.dev.register_scalars([a.numpy() for a in self.tracers], [a.numpy() for a in self.tend])
        if kind not in ("stage", "dropin"):
            self.dev.set_coherence(abi.RESIDENT)
        if kind == "window":
            self.dev.set_surface_emission(list(_emission(case).cpu().numpy()))
            self.lam, self.lam_tend = pinned((n, *w)), pinned((n, *w))

    def load(self, fields):
        """A new state into the host arrays that the library was given."""
        for k, x in fields.items():
            (self.arrays[k] if k in self.arrays else getattr(self, k)).copy_(x, non_blocking=True)
        torch.cuda.synchronize()


_model = (None, None)


def _model_of(case):
    global _model
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if _model[0] != key:
        if _model[1] is not None:
            _model[1].dev.close()
        _model = (None, None)
        _model = (key, _Model(case))
    return _model[1]


# ---- states ------------------------------------------------------------------

def _latlon(T, at):
    lat, lon = torch.deg2rad(T["glat" + at]), torch.deg2rad(T["glon" + at])
    return lat, lon


def _uniform(gen, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=gen, device=gen.device, dtype=torch.float64)


def _profile(T):
    """Temperature and pressure of a 6.5 K/km lapse rate from 300 K, held at 200 K above."""
    z = torch.linspace(0.0, float(T["zt"].max()) + 1.0, 4001, dtype=torch.float64)
    tz = torch.clamp(300.0 - 6.5e-3 * z, min=200.0)
    f = GRAV / (R_DRY * tz)
    lnp = math.log(P00) - torch.cat([torch.zeros(1, dtype=torch.float64),
                                     torch.cumsum(0.5 * (f[1:] + f[:-1]) * torch.diff(z), 0)])
    zt = T["zt"].cpu()
    p = torch.from_numpy(np.exp(np.interp(zt.numpy(), z.numpy(), lnp.numpy())))
    return torch.clamp(300.0 - 6.5e-3 * zt, min=200.0).to(T["zt"].device), p.to(T["zt"].device)


def _atmosphere(T, gen):
    """Seeded winds and thermodynamics: two mid-latitude jets of about
    35 m/s, theta perturbations of 0.5 K, vertical motion of a few cm/s."""
    temp, press = _profile(T)
    lat, lon = _latlon(T, "w")
    zt = T["zt"]
    pert = torch.zeros_like(T["volti"])
    for _ in range(3):
        a, b = _uniform(gen, -0.8, 0.8, 1), _uniform(gen, -math.pi, math.pi, 1)
        cosd = torch.sin(lat) * torch.sin(a) + torch.cos(lat) * torch.cos(a) * torch.cos(lon - b)
        r = ERAD * torch.arccos(torch.clamp(cosd, -1, 1))
        pert += 0.5 * torch.exp(-(r / 5.0e5) ** 2)[:, None] * torch.exp(-((zt - 5.0e3) / 3.0e3) ** 2)[None]
    theta = (temp * (P00 / press) ** (R_DRY / CP))[None] + pert
    rho = (press / float(ALPHA)) ** (CV / CP) / theta
    latv, lonv = _latlon(T, "v")
    prof = (torch.exp(-((latv.abs() - math.radians(45.0)) / math.radians(12.0)) ** 2)[:, None]
            * torch.exp(-((zt - 1.0e4) / 6.0e3) ** 2)[None])
    wave = 1.0 + 0.2 * torch.sin(4 * lonv + _uniform(gen, 0, 2 * math.pi, 1))
    east = T["vny"] * torch.cos(lonv) - T["vnx"] * torch.sin(lonv)
    vc = _uniform(gen, 30.0, 38.0, 1) * (wave * east)[:, None] * prof
    a = _uniform(gen, 0, 2 * math.pi, 3)
    horiz = torch.sin(3 * lon + a[0]) * torch.cos(2 * lat + a[1]) + 0.5 * torch.sin(5 * lon - a[2])
    wc = 0.05 * horiz[:, None] * torch.sin(math.pi * torch.clamp(T["zm"] / T["zm"][-1], 0, 1))[None]
    wc[:, 0] = wc[:, -1] = 0.0
    for x in (rho, theta, vc, wc):
        x[0] = 0.0
    return theta, rho, vc, wc


def _tracers(T, gen, case):
    """Lognormal mixing ratios around 1e-8 within 1e-12 .. 1e-6; every tenth
    tracer is zero above 15 km."""
    lat, lon = _latlon(T, "w")
    zt = T["zt"]
    out = torch.empty((case["ntr"], lat.numel(), zt.numel()), dtype=torch.float32, device=lat.device)
    for n in range(case["ntr"]):
        a, m = _uniform(gen, 0, 2 * math.pi, 3), torch.randint(1, 6, (2,), generator=gen, device=gen.device)
        h = torch.sin(m[0] * lon + a[0]) * torch.cos(m[1] * lat + a[1])
        h = h + 0.3 * torch.randn(h.shape, generator=gen, device=gen.device, dtype=torch.float64)
        v = 0.5 * torch.sin(2 * math.pi * zt / _uniform(gen, 5e3, 3e4, 1) + a[2])
        q = 1.0e-8 * torch.exp(1.25 * (h[:, None] + v[None]))
        q = torch.clamp(q, 1.0e-12, 1.0e-6)
        if n % 10 == 7:
            q[:, zt > 15000.0] = 0.0
        q = torch.where(T["open_w"], q, q.gather(1, T["kw"][:, None]))
        q[0] = 0.0
        out[n] = q.float()
    return out


def _emission(case):
    """A surface source per tracer [kg/kg/s x density], fixed for the run."""
    T = _tables_of(case)
    gen = torch.Generator(device=_device()).manual_seed(77)
    e = 1.0e-12 * torch.rand((case["ntr"], T["kw"].numel()), generator=gen, device=gen.device)
    e[:, 0] = 0.0
    return e


def _fields(case, seed):
    """The inputs of one pass, from the seed alone, on the device."""
    T = _tables_of(case)
    gen = torch.Generator(device=_device()).manual_seed(1000003 * seed + 17)
    theta, rho, vc, wc = _atmosphere(T, gen)
    iw1, iw2 = T["itab_v_iw"][:, 0], T["itab_v_iw"][:, 1]
    rhow = 0.5 * (rho + torch.roll(rho, -1, 1))
    f = {}
    if _dynamic(case):
        f["thil"] = theta.float()
        f["rho"] = rho
        f["press"] = float(ALPHA) * (rho * f["thil"].double()) ** (CP / CV)
        f["vc"], f["vmc"] = vc.float(), (vc * 0.5 * (rho[iw1] + rho[iw2])).float()
        f["wc"], f["wmc"] = wc.float(), (wc * rhow).float()
        wst = torch.cat([wc[:, :1], wc[:, :-1]], 1) + wc
        for n, x in enumerate(("vxe", "vye", "vze")):
            e = T[("wnxo2", "wnyo2", "wnzo2")[n]][:, None] * wst
            for j in range(7):
                e = e + T["ecvec_" + ("vx", "vy", "vz")[n]][:, j, None] * vc[T["itab_w_iv"][:, j]]
            e[:, 0], e[0] = e[:, 1], 0.0
            f[x] = e.float()
    else:
        vm = torch.where(T["open_v"], 0.5 * (rho[iw1] + rho[iw2]) * vc * T["arv"], 0.0).float()
        wm = torch.where(T["open_w"], wc * rhow * T["arw"], 0.0)
        wm[:, -1] = 0.0
        vm[0], wm[0] = 0.0, 0.0
        f["vmasc"], f["wmasc"], f["wc"], f["rho_old"] = vm, wm.float(), wc.float(), rho.float()
        f["rho"] = f["rho_old"].double() + _dt(case) * T["volti"] * _convergence(T, vm.double(), f["wmasc"].double())
        f["rho"] = torch.where(T["open_w"], f["rho"], f["rho_old"].double())
        f["rho"][0] = 0.0
    f["tracers"] = _tracers(T, gen, case)
    if case["kind"] in ("stage", "dropin"):   # tendencies of the host model's physics
        q = f["tracers"].double()
        tend = 1.0e-6 * q * torch.randn(q.shape[:2], generator=gen, device=gen.device, dtype=torch.float64)[..., None]
        f["tend"] = (tend * rho).float()
    if case["kind"] == "window":   # dJ/d(tracers) of receptors near the ground and aloft
        lam = torch.randn(f["tracers"].shape, generator=gen, device=gen.device)
        keep = torch.rand(lam.shape[1], generator=gen, device=gen.device) < 0.05
        keep[0] = False
        f["lam"] = torch.where(keep[None, :, None] & T["open_w"][None], lam, 0.0)
    return f


def prepare(case, seed):
    m, f = _model_of(case), _fields(case, seed)
    if case["kind"] == "stage":
        f = {k: f[k] for k in ("tracers", "tend", "rho", "vmasc", "wmasc")}
        scp = f["tracers"][0]
        f["rhos"] = f["rho"].float()
        f["scp0"] = (scp * (1.0 + 1.0e-3 * torch.sin(torch.arange(scp.shape[0], device=scp.device)))[:, None]).float()
        f["out"] = torch.zeros_like(scp)
    return dict(case=case, model=m, fields=f)


# ---- one pass ----------------------------------------------------------------

DYN_FIELDS = ("rho", "press", "thil", "wmc", "wc", "vmc", "vc", "vxe", "vye", "vze")
DYN_MASK = abi.F_RHO | abi.F_PRESS | abi.F_THIL | abi.F_WC | abi.F_WMC | abi.F_VXE | abi.F_VMC | abi.F_VC


def _split(x):
    """The tracers that exact() computes, and the others."""
    return dict(tracers=x[:EXACT_TRACERS], others=x[EXACT_TRACERS:]) if len(x) > EXACT_TRACERS else dict(tracers=x)


def run(state):
    case, m, f = state["case"], state["model"], state["fields"]
    kind, dev = case["kind"], m.dev
    if kind == "stage":
        p = lambda x: ctypes.c_void_p(x.data_ptr())  # noqa: E731
        check(dev.lib.olamgpu_update_scalar_noalloc(
            p(f["tracers"][0]), p(f["scp0"]), p(f["tend"][0]), p(f["rhos"]), p(f["vmasc"]), p(f["wmasc"]),
            ctypes.c_float(0.5 * _dt(case)), p(f["out"]), None))   # the library's stream
        return f["out"]
    m.load(f)
    if kind == "dropin":
        dev.scalar_transport_rk(m.rho_old.numpy())
        return _split(m.tracers.numpy())
    if not _dynamic(case):
        dev.sync_to_device(abi.F_SCALARS | abi.F_VMASC | abi.F_WMASC | abi.F_RHO | abi.F_WC)
        for n in range(case["steps"]):
            dev.scalar_transport_rk(None if n else m.rho_old.numpy())
        dev.sync_to_host(abi.F_SCALARS)
        return _split(m.tracers.numpy())
    dev.sync_to_device(DYN_MASK | abi.F_SCALARS)
    if kind == "long":
        for _ in range(case["steps"]):
            dev.timestep(abi.TS_GRAPH)
        dev.sync_to_host(DYN_MASK | abi.F_SCALARS)
        return {k: m.arrays[k].numpy() for k in DYN_FIELDS} | _split(m.tracers.numpy())
    dev.window_forward(case["steps"], 4, abi.TS_GRAPH)
    dev.sync_to_host(abi.F_SCALARS)
    dev.window_adjoint([x.numpy() for x in m.lam], [x.numpy() for x in m.lam_tend], in_place=True)
    return dict(tracers=m.tracers.numpy(), grad=m.lam.numpy(), grad_tend=m.lam_tend.numpy())


# ---- what a pass cannot do without ---------------------------------------------

def work(case):
    """Bytes and operations per pass: for each RK stage of a tracer its
    input, start value and tendency read and the result written (stage 1's
    input is the start value), the winds, densities and volumes once per
    stage; for each acoustic stage the state, its start values and the
    metric arrays read and the state written."""
    nxp, cells = case["nxp"], (10 * case["nxp"] ** 2 + 2) * case["nlev"]
    ntr, nrk, wind = case["ntr"], case["nrk"], 32.0
    per = 90.0 if case["order"] == 2 else 150.0
    if case["kind"] == "stage":
        return dict(bytes=cells * (16 + 24.0), flops=cells * per)
    step_b = cells * (ntr * (12.0 + 16.0 * (nrk - 1)) + nrk * wind)
    step_f = cells * ntr * nrk * per
    if case["kind"] == "limited":
        step_f *= 1.5
    if not _dynamic(case):
        return dict(bytes=case["steps"] * step_b, flops=case["steps"] * step_f)
    core_b = cells * NACOUST * (3 * 208.0 + 80.0)
    core_f = cells * NACOUST * 3 * 700.0
    n = case["steps"]
    if case["kind"] == "long":
        return dict(bytes=n * (step_b + core_b), flops=n * (step_f + core_f))
    back = cells * ntr * 24.0 * nrk
    return dict(bytes=n * (step_b + back + 2 * core_b), flops=n * (2 * step_f + 2 * core_f))


# ---- the same in 64 bits ---------------------------------------------------------

def _convergence(T, vm, wm):
    """Mass flux convergence of every cell: edges and the two W faces."""
    d = torch.cat([wm[:, :1], wm[:, :-1]], 1) * (torch.arange(wm.shape[1], device=wm.device) > 0) - wm
    for n in range(7):
        d = d + T["dirv"][:, n, None] * vm[T["itab_w_iv"][:, n]]
    return d


def _shift(x, up):
    """Level k-1 (up=False) or k+1 of x at level k; the end level repeats."""
    return torch.cat([x[:, 1:], x[:, -1:]], 1) if up else torch.cat([x[:, :1], x[:, :-1]], 1)


class _Transport:
    """One stage of update_scalar (every column explicit) for given winds."""

    def __init__(self, case, vm, wm, rhos):
        self.T = T = _tables_of(case)
        self.order = case["order"]
        self.vm, self.wm, self.rhos = torch.where(T["open_v"], vm, 0.0), wm, rhos
        lev = torch.arange(wm.shape[1], device=wm.device)[None]
        kw = T["kw"][:, None]
        self.kw, self.top = kw, wm.shape[1] - 1
        self.below, self.at_top, self.floor = lev == kw - 1, lev == self.top, lev == kw
        self.open = T["open_w"]
        wmm = _shift(wm, False) * (lev > 0)
        self.wm0, self.wm1 = wmm, wm
        self.net = _convergence(T, self.vm, wm)
        self.scale = torch.where(self.open & (rhos != 0), T["volti"] / torch.where(rhos == 0, 1.0, rhos), 0.0)
        self.inv = torch.where(self.open & (rhos != 0), 1.0 / torch.where(rhos == 0, 1.0, rhos), 0.0)
        self.ev = T["itab_w_iv"]
        self.iw1, self.iw2 = T["itab_v_iw"][:, 0], T["itab_v_iw"][:, 1]
        self.faces = [T["open_v"][self.ev[:, n]] & T["valid"][:, n, None] for n in range(7)]

    def face_v(self, s, unbounded=False):
        """Upwind reconstruction at the V faces (order 2 or 3)."""
        T = self.T
        if self.order == 2:
            w, c = [T["gxps_coef"], T["gyps_coef"]], [T["dxps"], T["dyps"]]
        else:
            xy, u = T["xy_hu" if unbounded else "xy_h"], "u" if unbounded else ""
            w = [xy[:, :, m] for m in range(5)]
            c = [T["dxps"], T["dyps"], T["xx0_v" + u], T["xy0_v" + u], T["yy0_v" + u]]
        planes = [torch.zeros_like(s) for _ in w]
        for n in range(7):
            d = torch.where(self.faces[n], s[T["itab_w_iw"][:, n]] - s, 0.0)
            planes = [p + x[:, n, None] * d for p, x in zip(planes, w)]
        side = [s[i] + sum(x[:, j, None] * p[i] for x, p in zip(c, planes))
                for j, i in enumerate((self.iw1, self.iw2))]
        return torch.where(self.vm < 0, side[1], side[0])

    def face_w(self, s, unbounded=False):
        """(value from below, value from above) at the top face of a level."""
        a = self.T["a_wu" if unbounded else "a_w"]
        up = torch.where(self.open & ~self.at_top, _shift(s, True) - s, 0.0)
        dn = torch.where(self.open & ~self.floor, s - _shift(s, False), 0.0)
        if unbounded:
            dn = torch.where(self.floor, up, dn)
            up = torch.where(self.at_top, dn, up)
        bot = s + up * a[0, 0][None] + dn * a[1, 0][None]
        top = s + up * a[0, 1][None] + dn * a[1, 1][None]
        return top, _shift(bot, True)

    def upwind_w(self, s):
        top, bot = self.face_w(s)
        v = torch.where(self.wm < 0, bot, top)
        v = torch.where(self.below, _shift(s, True), v)
        return torch.where(self.at_top, s, v)

    def flux(self, up_v, up_w):
        f = self.vm * up_v
        d = self.wm0 * _shift(up_w, False) - self.wm1 * up_w
        for n in range(7):
            d = d + self.T["dirv"][:, n, None] * f[self.ev[:, n]]
        return d

    def fill(self, new, rest):
        """Levels under ground take the floor's value, the dummy column keeps its own."""
        new = torch.where(self.open, new, new.gather(1, self.kw.expand(-1, 1)))
        return torch.cat([rest[:1], new[1:]])

    def stage(self, s, s0, tend, dtr):
        d = self.flux(self.face_v(s), self.upwind_w(s)) - self.net * s0
        return self.fill(s0 + dtr * (self.inv * tend + self.scale * d), s0)

    def limited(self, s, s0, dtr, monot):
        """The flux-corrected last stage (flat grid, no tendency)."""
        T, vm, wm = self.T, self.vm, self.wm
        e0, e1 = float(np.float32(1e-32)), float(np.float32(3e-7))
        neg, iw1, iw2 = vm < 0, self.iw1, self.iw2
        lo_v = torch.where(neg, s0[iw2], s0[iw1])
        hi_v = self.face_v(s, monot) - lo_v
        f_v = vm * hi_v
        inner = self.open & ~self.at_top
        lo_w = torch.where(wm < 0, _shift(s0, True), s0)
        end = s0 if monot else s
        lo_w = torch.where(self.below, _shift(end, True), torch.where(self.at_top, end, lo_w))
        top, bot = self.face_w(s, monot)
        hi_w = torch.where(inner, torch.where(wm < 0, bot, top) - lo_w, 0.0)
        f_w = wm * hi_w
        f_wm = torch.where(self.open & ~self.floor, _shift(f_w, False), 0.0)
        low = self.flux(lo_v, lo_w) - self.net * s0
        fin, fout = f_wm.clamp(min=0) - f_w.clamp(max=0), f_wm.clamp(max=0) - f_w.clamp(min=0)
        big, small = s0.clone(), s0.clone()
        from_below = self.open & ~self.floor & (self.wm0 > 0)
        from_above = inner & (wm < 0)
        for m, x in ((from_below, _shift(s0, False)), (from_above, _shift(s0, True))):
            big, small = torch.where(m, torch.maximum(big, x), big), torch.where(m, torch.minimum(small, x), small)
        for n in range(7):
            e = T["dirv"][:, n, None] * f_v[self.ev[:, n]]
            fin, fout = fin + e.clamp(min=0), fout + e.clamp(max=0)
            if monot:
                x = s0[T["itab_w_iw"][:, n]]
                m = self.faces[n] & (T["dirv"][:, n, None] * vm[self.ev[:, n]] > 0)
                big, small = torch.where(m, torch.maximum(big, x), big), torch.where(m, torch.minimum(small, x), small)
        rh, vt = self.rhos, T["volti"]
        q = s0 * rh + dtr * vt * low
        if monot:
            d = (1 + e1) * dtr * vt
            a_in = (rh * big - (q + e1 * q.abs()) - e0).clamp(min=0)
            a_out = (rh * small - (q - e1 * q.abs()) + e0).clamp(max=0)
            r_in = (a_in / torch.maximum((d * fin).clamp(min=e0), 0.01 * a_in)).clamp(max=1)
            r_out = (a_out / torch.minimum((d * fout).clamp(max=-e0), 0.01 * a_out)).clamp(max=1)
            c_w = torch.where(f_w < 0, torch.minimum(r_in, _shift(r_out, True)),
                              torch.minimum(_shift(r_in, True), r_out))
            c_v = torch.where(f_v < 0, torch.minimum(r_in[iw1], r_out[iw2]), torch.minimum(r_in[iw2], r_out[iw1]))
        else:
            a_out = ((1 - e1) * q - e0).clamp(min=0)
            r = (a_out / torch.maximum((-(1 + e1) * dtr * vt * fout).clamp(min=e0), 0.01 * a_out)).clamp(max=1)
            c_w = torch.where(f_w < 0, _shift(r, True), r)
            c_v = torch.where(f_v < 0, r[iw2], r[iw1])
        d = self.flux(lo_v + hi_v * c_v, lo_w + torch.where(inner, hi_w * c_w, 0.0)) - self.net * s0
        new = s0 + dtr * self.scale * d
        new[:, 0] = s[:, 0]
        return torch.cat([s0[:1], new[1:]])

    def step(self, q, tend, case):
        """scalar_transport_rk of one tracer."""
        dt, nrk = _dt(case), case["nrk"]
        s = q
        for n, x in enumerate((1.0 / 3.0, 0.5, 1.0) if nrk == 3 else (0.5, 1.0)):
            if n == nrk - 1 and case["monot"]:
                s = self.limited(s, q, x * dt, case["monot"] == 1)
            else:
                s = self.stage(s, q, tend, x * dt)
        return s


class _Core:
    """The dynamical core's long step (flat grid, dry, second order)."""

    def __init__(self, case, f):
        self.case, self.T = case, _tables_of(case)
        self.opts = abi.make_opts(_dt(case), nacoust=NACOUST, nrk_scal=case["nrk"])
        self.s = {k: f[k].double().clone() for k in DYN_FIELDS}
        T = self.T
        self.open_w, self.open_v = T["open_w"], T["open_v"]
        nz = self.open_w.shape[1]
        self.lev = torch.arange(nz, device=self.open_w.device)[None]
        self.inner = self.open_w & (self.lev < nz - 1)
        self.iw1, self.iw2 = T["itab_v_iw"][:, 0], T["itab_v_iw"][:, 1]
        self.pwfac = T["dzim"][None].float().double()
        self.pvfac = (T["zfacit"][None].float() * T["dniv"][:, None].float()).double()
        o, im = self.opts, T["itab_v_im"]
        iv = T["itab_m_iv"]
        second = torch.stack([im[iv[:, j], 1] == torch.arange(iv.shape[0], device=iv.device) for j in range(3)], 1)
        arm0 = torch.where(T["arm0"] == 0, 1.0, T["arm0"])
        v = T["dnv"][iv] / arm0[:, None]
        self.vfact = torch.where(second, v, -v)
        amin = torch.minimum(T["arw0"][self.iw1], T["arw0"][self.iw2])
        vmin = torch.minimum(T["volt"][self.iw1], T["volt"][self.iw2])
        f = float(np.float32(o.divh_damp_fact))
        self.fdiv = (f ** 3 / o.dtsm * amin ** 2 * T["dniv"])[:, None] * (T["zfacit"] * T["dzit"])[None] * vmin
        a = -float(np.float32(o.vort_damp_fact)) * torch.minimum(T["arm0"][im[:, 0]], T["arm0"][im[:, 1]])
        self.fvor = (0.5 * T["dniu"] / o.dtsm * a ** 3)[:, None]

    def damping(self):
        T, s = self.T, self.s
        d = torch.zeros_like(s["rho"])
        for n in range(7):
            i = T["itab_w_iv"][:, n]
            d = d - T["dirv"][:, n, None] * (T["arv"] * s["vmc"])[i]
        d = torch.where(self.open_w, d * T["volti"], 0.0)
        for _ in range(2):
            x = sum((d[T["itab_w_iw"][:, n]] - d) * (T["xx_yy"][:, n] * T["valid"][:, n])[:, None] for n in range(7))
            d = torch.where(self.open_w, x, 0.0)
            d[0] = 0.0
        t = self.fdiv * (d[self.iw2] - d[self.iw1])
        v = sum(s["vc"][T["itab_m_iv"][:, j]] * self.vfact[:, j, None] for j in range(3))
        v = torch.where(self.lev >= 1, v, 0.0)
        for _ in range(2):
            x = sum((v[T["itab_m_im"][:, j]] - v) * T["xx_yy_m"][:, j, None] for j in range(3))
            v = torch.where(self.lev >= 1, x, 0.0)
            v[0] = 0.0
        im = T["itab_v_im"]
        t = t + self.fvor * (v[im[:, 1]] - v[im[:, 0]]) * (s["rho"][self.iw1] + s["rho"][self.iw2])
        return torch.where(self.open_v, t, 0.0)

    def acoustic(self, vmasc, wmasc):
        T, s, o = self.T, self.s, self.opts
        rho0, rth0, wmc0, vmc0 = s["rho"].clone(), s["rho"] * s["thil"], s["wmc"].clone(), s["vmc"].clone()
        short = self.damping()
        fr = float(np.float32(0.70))
        pc = fr * float(np.float32(1004.0) / np.float32(717.0))
        rocv = float((np.float32(1004.0) - np.float32(717.0)) / np.float32(717.0))
        wn = [T[k][:, None] for k in ("wnx", "wny", "wnz")]
        for st, x in enumerate((1.0 / 3.0, 0.5, 1.0)):
            dt = x * o.dtsm
            flow = _Transport(self.case | {"order": 2}, s["vmc"] * T["arv"], s["wmc"], torch.ones_like(s["rho"]))
            if st == 2:
                vmasc += torch.where(self.open_v, flow.vm, 0.0)
            four = [s[k] for k in ("thil", "vxe", "vye", "vze")]
            up_w = [flow.upwind_w(q) for q in four]
            hsum = [torch.zeros_like(rho0) for _ in range(5)]
            fv = [flow.vm] + [flow.vm * flow.face_v(q) for q in four]
            for n in range(7):
                i, dv = T["itab_w_iv"][:, n], T["dirv"][:, n, None]
                hsum = [h + dv * q[i] for h, q in zip(hsum, fv)]
            hf, th, rk = hsum[0], hsum[1], hsum[2:]
            mass = s["rho"] * T["volt"]
            fc = float(o.fcoriol)
            rk = [rk[0] + mass * fc * s["vye"], rk[1] - mass * fc * s["vxe"], rk[2]]
            rt = s["rho"] * s["thil"]
            b10 = dt * T["volti"]
            b5 = float(ALPHA) * torch.where(rt > 0, rt, 1.0) ** rocv
            drho, drt = b10 * hf, b10 * th
            if st:
                drho, drt = drho + rho0 - s["rho"], drt + rth0 - rt
            pex, rex, b15 = b5 * (rt + pc * drt), s["rho"] + fr * drho, b10 * b5
            up = lambda q: _shift(q, True)  # noqa: E731
            vi = T["volwi"]
            dwm = wmc0 + dt * ((pex - up(pex)) * self.pwfac - (T["gdz_wgtm8"] * rex + T["gdz_wgtp8"] * up(rex))
                               + sum(w * (q + up(q)) for w, q in zip(wn, rk)) * vi)
            b7, b8, c9 = dt * vi, dt * pc * self.pwfac, -dt * dt * fr
            b21, b22 = b7 * _shift(s["wc"], False), b7 * up(s["wc"])
            b23, b24 = b8 * b15, b8 * up(b15)
            b25, b26 = c9 * T["volti"] * T["gdz_wgtm"], c9 * up(T["volti"]) * T["gdz_wgtp"]
            tw = up_w[0]
            lo = -_shift(T["arw"], False) * (b21 + b25 + b23 * _shift(tw, False))
            di = 1.0 + T["arw"] * (b25 - b26 + (b23 + b24) * tw)
            hi = up(T["arw"]) * (b22 + b26 - b24 * up(tw))
            w = self.solve(lo, di, hi, dwm)
            wma = torch.where(self.inner, w * T["arw"], 0.0)
            if st == 2:
                wmasc += wma
            below = lambda q: torch.where(self.lev > 1, _shift(q, False), 0.0)  # noqa: E731
            net = lambda q: below(q) - q  # noqa: E731
            rho = rho0 + b10 * (hf + net(wma))
            drt = drt + b10 * net(wma * tw)
            rk = [q + net(wma * u) for q, u in zip(rk, up_w[1:])]
            safe = torch.where(rho == 0, 1.0, rho)
            self.put("rho", rho)
            self.put("press", b5 * (rt + pc * drt))
            self.put("thil", (rt + drt) / safe, ground=True)
            zw = T["zwgt_bot8"] * safe + T["zwgt_top8"] * up(safe)
            s["wmc"][1:] = torch.where(self.inner, w, s["wmc"])[1:]
            wc = torch.where(self.inner, w / zw, s["wc"])
            wc[:, 0] = wc[:, 1]
            s["wc"][1:] = wc[1:]
            vn = [T[k][:, None] for k in ("vnx", "vny", "vnz")]
            pg = (s["press"][self.iw1] - s["press"][self.iw2]) * self.pvfac
            force = sum(c * (q[self.iw1] + q[self.iw2]) for c, q in zip(vn, rk)) * T["volvi"]
            v = vmc0 + dt * (short + pg + force)
            two = s["rho"][self.iw1] + s["rho"][self.iw2]
            for k, q in (("vmc", v), ("vc", 2.0 * v / torch.where(two == 0, 1.0, two))):
                s[k][1:] = torch.where(self.open_v, q, s[k])[1:]
            wst = _shift(s["wc"], False) + s["wc"]
            for k, wo, e in (("vxe", "wnxo2", "ecvec_vx"), ("vye", "wnyo2", "ecvec_vy"), ("vze", "wnzo2", "ecvec_vz")):
                q = wst * T[wo][:, None]
                for n in range(7):
                    q = q + (T[e][:, n] * T["valid"][:, n])[:, None] * s["vc"][T["itab_w_iv"][:, n]]
                self.put(k, q, ground=True)

    def put(self, k, x, ground=False):
        x = torch.where(self.open_w, x, x[:, 1:2] if ground else self.s[k])
        self.s[k][1:] = x[1:]

    def solve(self, lo, di, hi, d):
        """The tridiagonal W system of levels 1 .. top - 1, by elimination."""
        top = d.shape[1] - 1
        g, x = [None] * (top + 1), [None] * (top + 1)
        c, y = None, None
        for k in range(1, top):
            den = di[:, k] - (lo[:, k] * c if k > 1 else 0.0)
            den = torch.where(den == 0, 1.0, den)
            y = (d[:, k] - (lo[:, k] * y if k > 1 else 0.0)) / den
            c = hi[:, k] / den
            g[k], x[k] = c, y
        for k in range(top - 2, 0, -1):
            x[k] = x[k] - g[k] * x[k + 1]
        out = torch.zeros_like(d)
        out[:, 1:top] = torch.stack(x[1:top], 1)
        return out

    def long_step(self):
        """Advances the core; returns the transport's winds and densities."""
        rho_old = self.s["rho"].clone()
        vmasc, wmasc = torch.zeros_like(self.s["vmc"]), torch.zeros_like(rho_old)
        for _ in range(NACOUST):
            self.acoustic(vmasc, wmasc)
        wmasc = torch.where(self.inner, wmasc / NACOUST, 0.0)
        return _Transport(self.case, vmasc / NACOUST, wmasc, self.s["rho"].clone())


def exact(case, seed):
    T, f = _tables_of(case), _fields(case, seed)
    n = min(case["ntr"], EXACT_TRACERS)
    more = {"others": None} if case["ntr"] > EXACT_TRACERS else {}
    with torch.no_grad():
        if not _dynamic(case):
            rhos = f["rho"]
            tr = _Transport(case, f["vmasc"].double(), f["wmasc"].double(),
                            rhos.float().double() if case["kind"] == "stage" else rhos)
            if case["kind"] == "stage":
                scp = f["tracers"][0]
                s0 = (scp * (1.0 + 1.0e-3 * torch.sin(torch.arange(scp.shape[0], device=scp.device)))[:, None]).float()
                out = tr.stage(scp.double(), s0.double(), f["tend"][0].double(), 0.5 * _dt(case))
                return torch.cat([torch.zeros_like(out[:1]), out[1:]])   # the dummy column is not written
            out = torch.empty((n, *rhos.shape), dtype=torch.float64, device=rhos.device)
            for i in range(n):
                q = f["tracers"][i].double()
                tend = f["tend"][i].double() if "tend" in f else torch.zeros_like(q)
                for _ in range(case["steps"]):
                    q = tr.step(q, tend, case)
                out[i] = q
            return dict(tracers=out, **more)
        core = _Core(case, f)
        q = [f["tracers"][i].double() for i in range(n if case["kind"] == "long" else case["ntr"])]
        emis = _emission(case).double() if case["kind"] == "window" else None
        tend = [torch.zeros_like(x) for x in q]
        if emis is not None:
            for i, t in enumerate(tend):
                t[:, 1] = emis[i]
        flows = []
        for _ in range(case["steps"]):
            tr = core.long_step()
            q = [tr.step(x, t, case) for x, t in zip(q, tend)]
            if emis is not None:
                flows.append(tr)
        if case["kind"] == "long":
            return {k: core.s[k] for k in DYN_FIELDS} | dict(tracers=torch.stack(q), **more)
    grad, grad_tend = torch.empty_like(torch.stack(q)), torch.zeros_like(torch.stack(q))
    for i in range(len(q)):
        lam = f["lam"][i].double()
        for tr in reversed(flows):
            # the step is linear in the tracer and its tendency: any point will do
            x, t = (torch.zeros_like(lam).requires_grad_() for _ in range(2))
            lam, g = torch.autograd.grad(tr.step(x, t, case), (x, t), lam)
            grad_tend[i] += g
        grad[i] = lam
    return dict(tracers=torch.stack(q), grad=grad, grad_tend=grad_tend)
