"""What a user of this framework has it do, as cases that can be timed.

A case is a dict of plain values; `prepare` makes the user's side of it (the
gas field and sources from a seed, a context with the particles loaded and
the octree built, rays where the caller makes its own, pinned buffers for
the results), `run` is one pass through the public entry points, `work` what
such a pass cannot do without. Kinds:

  ticks   batches of ticks on one field and the particle state read back, as
          an epoch does between two outputs. `emit`: the rays come from the
          library's own sources (psg_run_ticks_emit, the C driver's way),
          else from the caller's host memory (psg_run_ticks). Physics:
          isothermal or not, hydrogen or with helium and secondary
          ionisation, on the spot or with recombination rays.
  trace   hit lists of a batch of rays on the host (psg_trace)
  epoch   an epoch's switch: particles loaded, octree built, first rays
          traced (psg_load_particles, psg_build_tree, psg_trace)
  steps   a host's own particle steps (psg_step_evolve)
  train   optimiser steps of the chemistry network (psg_mlp_grad,
          psg_mlp_adam)

Successive passes go on in simulated time, as a run does: the gas ionises
and the sources emit new rays from pass to pass.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from psphray_b200 import api, fields
from psphray_b200.surrogate import NFEAT, NPARAM, init_params
from psphray_b200.units import Units

DEV = "cuda:0"
NGB = 32                    # neighbours inside a smoothing length
TICK_MYR = 0.05             # 500 Myr in 10,000 ticks
HOST_BATCHES = 4            # ray batches a host-side caller has at hand


def listed() -> list:
    ticks = dict(kind="ticks", calls=1, sigma=1.0, nsrc=16, emit=True, iso=False, helium=False, on_the_spot=True)
    uniform = dict(ticks, sigma=0.0, nsrc=1, iso=True)
    return [
        # the reference's CPU-sized run, stepped tick by tick by a host that
        # makes its own rays: nothing but latency and launches
        dict(uniform, name="uniform32_tick", side=32, rays=32, ticks=1, emit=False),
        # the 64^3 uniform field with one corner source, isothermal, in
        # batches of 100 ticks: many short ticks in one call
        dict(uniform, name="uniform64", side=64, rays=1024, ticks=100),
        # the benchmark's field: 2M particles, log-normal, 16 sources, not
        # isothermal, 8 ticks to a call
        dict(ticks, name="lognormal128", side=128, rays=8192, ticks=8),
        # the full pipeline's field: 16.8M particles, 256 sources, 65536 rays
        # per tick, called tick by tick
        dict(ticks, name="lognormal256", side=256, rays=65536, ticks=1, calls=4, sigma=1.5, nsrc=256),
        # sizes nobody chose for the machine: 45^3 particles, 777 rays from
        # host memory, 7 ticks
        dict(ticks, name="lognormal45_host", side=45, rays=777, ticks=7, nsrc=5, emit=False),
        # recombination rays (not on the spot): ticks depend on one another
        dict(ticks, name="recombination100", side=100, rays=3000, ticks=6, on_the_spot=False),
        # helium and secondary ionisation on the spot, the benchmark's field
        dict(ticks, name="helium128", side=128, rays=8192, ticks=4, helium=True),
        # the reference's default physics together: helium, secondary
        # ionisation, recombination rays, not isothermal
        dict(ticks, name="default_physics64", side=64, rays=1024, ticks=8, helium=True, on_the_spot=False),
        # hit lists for a host that does its own deposit: trace()
        dict(kind="trace", name="trace64", side=64, sigma=0.0, rays=1024),
        # rt_switch_epoch() of the benchmark's field and its first rays
        dict(kind="epoch", name="epoch128", side=128, sigma=1.0, rays=64),
        # step_evolve() for a host that keeps the particles itself
        dict(kind="steps", name="steps30000", n=30000, iso=False),
        # the chemistry network's training at the shipped batch size
        dict(kind="train", name="train8192", batch=8192, steps=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    u = rng.random()
    if u < 0.68:
        physics = rng.choice(["iso", "hydrogen", "hydrogen", "recombination", "helium", "default"])
        sigma = 0.0 if physics == "iso" else rng.choice([1.0, 1.0, 1.5])
        side = _log_int(rng, 20, 150)
        per_ray = _hits_per_ray(side, sigma)
        rays = _log_int(rng, 24, 12000)
        most = 3e7 / (1 if physics in ("iso", "hydrogen") else 4)
        ticks = _log_int(rng, 1, max(1, min(64, int(most / (rays * per_ray)), int(2.5e8 / side ** 3))))
        return dict(kind="ticks", side=side, rays=rays, ticks=ticks, calls=1, sigma=sigma,
                    nsrc=1 if sigma == 0.0 else _log_int(rng, 1, 64),
                    emit=physics not in ("iso", "hydrogen") or rng.random() < 0.6, iso=physics == "iso",
                    helium=physics in ("helium", "default"), on_the_spot=physics not in ("recombination", "default"))
    if u < 0.78:
        return dict(kind="trace", side=_log_int(rng, 20, 150), sigma=rng.choice([0.0, 1.0]), rays=_log_int(rng, 1, 4000))
    if u < 0.86:
        return dict(kind="epoch", side=_log_int(rng, 20, 150), sigma=rng.choice([0.0, 1.0]), rays=_log_int(rng, 1, 100))
    if u < 0.94:
        return dict(kind="steps", n=_log_int(rng, 1, 60000), iso=rng.random() < 0.5)
    return dict(kind="train", batch=_log_int(rng, 100, 16384), steps=rng.randint(1, 8))


# ---- the user's side ---------------------------------------------------------
def _field(side, sigma, units, seed) -> fields.Field:
    """side^3 equal-mass particles, uniform (sigma 0) or placed by mass on
    exp(sigma*g), g a Gaussian random field of spectrum k^-2, like
    fields.uniform_field and lognormal_field; the smoothing length is that
    of the density around the particle's cell with the scatter that the
    distance to the 32nd of Poisson neighbours has (a neighbour search of
    millions of particles would take longer than everything that is timed)."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    n = side ** 3
    box = 6.6 * units.KPC
    rand = torch.rand((n, 3), generator=gen, device=DEV, dtype=torch.float64)
    if sigma > 0.0:
        k = torch.fft.fftfreq(side, device=DEV) * side
        kz = torch.fft.rfftfreq(side, device=DEV) * side
        k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2
        k2[0, 0, 0] = 1.0
        amp = k2.rsqrt()
        amp[0, 0, 0] = 0.0
        g = torch.fft.irfftn(torch.fft.rfftn(torch.randn((side,) * 3, generator=gen, device=DEV)) * amp, s=(side,) * 3)
        dens = torch.exp(sigma * ((g - g.mean()) / g.std()).double() - 0.5 * sigma * sigma).reshape(-1)
        dens /= dens.mean()
        cdf = (dens * 2.0 ** 24).long().cumsum(0)      # whole numbers: the same sums every time
        u = (torch.rand(n, generator=gen, device=DEV, dtype=torch.float64) * cdf[-1]).long()
        cell = torch.searchsorted(cdf, u, right=True).clamp_max(n - 1)
        ijk = torch.stack([cell // (side * side), cell // side % side, cell % side], 1)
        pos = ((ijk + rand) * (box / side)).float()
        rel = dens[cell]
        around = torch.nn.functional.pad(dens.view(1, 1, side, side, side), (1,) * 6, mode="circular")
        around = torch.nn.functional.avg_pool3d(around, 3, 1).reshape(-1)[cell]
    else:
        pos = (rand * box).float()
        rel = around = torch.ones(n, device=DEV, dtype=torch.float64)
    pos = pos.clamp_max(float(np.nextafter(np.float32(box), np.float32(0))))
    mass = 1e-3 * (box / units.CM) ** 3 / n / units.H_PER_MASS      # one hydrogen atom per 1000 cm^3
    z = torch.randn(n, generator=gen, device=DEV)
    sml = (3.0 * NGB / (4.0 * math.pi * n * around)).pow(1.0 / 3.0).float() * box * (1.0 - 1.0 / (9 * NGB) + z / (3 * NGB ** 0.5))
    full = lambda v: np.full(n, v, np.float32)      # noqa: E731
    xHII = 1.2e-3
    ye = xHII + (0.25 * units.hemf / units.hmf * 0.1 if units.hemf > 0 else 0.0)
    return fields.Field(pos=pos.cpu().numpy(), mass=full(mass), sml=sml.float().cpu().numpy(),
                        rho=(rel * (mass * n / box ** 3)).float().cpu().numpy(), ie=full(units.Tye2ie(1e4, xHII)),
                        xHI=full(1.0 - xHII), ye=full(ye), boxsize=float(box), units=units)


def _sources(case, units, boxsize, seed):
    """The sources and their spectrum: one in the corner (5e48 photons/s at
    13.6 eV), or nsrc random ones (1e47 to 1e49, from 1e46 on the wider
    field) with an 8-line 1e5 K blackbody."""
    if case["sigma"] == 0.0:
        src = [fields.Source(pos=(0.0, 0.0, 0.0), ngamma_dot=5e48 / units.SEC)]
        return src, (np.array([13.6 * units.EV]), np.array([1.0]))
    rng = np.random.default_rng(seed)
    pos = rng.random((case["nsrc"], 3)) * boxsize
    lum = 10 ** rng.uniform(47 if case["sigma"] < 1.5 else 46, 49, case["nsrc"])
    return ([fields.Source(pos=tuple(p), ngamma_dot=float(v) / units.SEC) for p, v in zip(pos, lum)],
            fields.blackbody_bins(units))


def _pinned(n, dtype):
    return torch.empty(n, dtype=dtype, pin_memory=True).numpy()


class HitList:
    """A host's own growing array of hits, as the reference's rt_trace()
    keeps one: malloc'd, handed to psg_trace() call after call."""

    def __init__(self, capacity):
        libc = C.CDLL(None)
        libc.calloc.restype = C.c_void_p
        self.free = libc.free
        self.size = C.c_size_t(capacity)
        self.x = C.c_void_p(libc.calloc(C.c_size_t(capacity), C.c_size_t(api.XTYPE_DTYPE.itemsize)))

    def array(self):
        raw = (C.c_char * (self.size.value * api.XTYPE_DTYPE.itemsize)).from_address(self.x.value)
        raw.owner = self        # the list lives as long as a view of it
        return np.frombuffer(raw, api.XTYPE_DTYPE)

    def __del__(self):
        self.free(self.x)


def prepare(case, seed) -> dict:
    if case["kind"] == "steps":
        return _prepare_steps(case, seed)
    if case["kind"] == "train":
        return _prepare_train(case, seed)
    helium = case.get("helium", False)
    units = Units(hmf=0.76 if helium else 1.0)
    f = _field(case["side"], case["sigma"], units, seed)
    ctx = api.Context(0)
    ctx.set_physics(api.Physics(units, isothermal=case.get("iso", True), h_only=not helium,
                                secondary_ionization=helium, on_the_spot=case.get("on_the_spot", True)))
    s = dict(case, ctx=ctx, tick_time=TICK_MYR * units.MYR, tick=1)
    case = dict(case, nsrc=case.get("nsrc", 16))
    sources, (eng, weight) = _sources(case, units, f.boxsize, seed + 1)
    if case["kind"] in ("trace", "epoch"):
        s["list"] = HitList(2 * int(case["rays"] * _hits_per_ray(case["side"], case["sigma"])) + 8 * case["side"])
    if case["kind"] == "epoch":
        s["field"] = f
    else:
        ctx.load(f)
        ctx.build_tree(8)
    if case["kind"] != "ticks" or not case["emit"]:
        T = case.get("ticks", 1)
        sch = fields.RaySchedule(sources=sources, nray=case["rays"], tick_time=s["tick_time"], boxsize=f.boxsize,
                                 seed=seed + 2, energies=eng, eweights=weight)
        s["rays"] = [sch.rays_for_ticks(1 + b * T, T) for b in range(HOST_BATCHES)]
    if case["kind"] == "ticks":
        if case["emit"]:
            ctx.set_sources(sources, [(eng, weight)], seed=seed + 2)
        if not case["on_the_spot"]:
            ctx.set_recombination(nrec=100, seed=seed + 3)
        n = f.n
        s["out"] = {"lambdaH": _pinned(n, torch.float64), "ie": _pinned(n, torch.float32),
                    "hits": _pinned(n, torch.int32), "lasthit": _pinned(n, torch.int64)}
        if helium:
            s["he"] = {"lambdaHeI": _pinned(n, torch.float64), "lambdaHeII": _pinned(n, torch.float64)}
    torch.cuda.empty_cache()
    return s


def _prepare_steps(case, seed) -> dict:
    """Records as update_pars() makes them: neutral to ionised particles of
    a log-normal density, most of them hit, over 1 to 200 ticks."""
    units = Units(hmf=1.0)
    ctx = api.Context(0)
    ctx.set_physics(api.Physics(units, isothermal=case["iso"]))
    return dict(case, ctx=ctx, records=_step_records(case, units, seed))


def _step_records(case, units, seed) -> np.ndarray:
    rng = np.random.default_rng(seed)
    n = case["n"]
    r = np.zeros(n, api.STEP_DTYPE)
    r["lambdaH"] = 10 ** rng.uniform(-6, 0, n)
    ie0 = units.Tye2ie(1e4, 1.2e-3)
    r["ie"] = ie0 * 10 ** rng.uniform(-0.5, 0.5, n)
    r["yGdepHI"] = np.where(rng.random(n) < 0.7, 10 ** rng.uniform(-4, 0, n), 0.0) * r["lambdaH"]
    r["heat"] = r["yGdepHI"] * 1e-3 * ie0
    r["time"] = TICK_MYR * units.MYR * rng.integers(1, 201, n)
    r["nH"] = 1e-3 / units.CM ** 3 * np.exp(rng.normal(0.0, 1.0, n))
    r["T"] = units.MPROTON_OVER_BOLTZMANN * r["ie"] / (1.0 + (1.0 - r["lambdaH"])) * 2.0 / 3.0
    return r


def _train_inputs(case, seed):
    """Normalised inputs and a smooth target, weights and Adam's moments in
    the middle of a run (step 200)."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    rows = case["batch"] * 16
    X = torch.zeros((rows, 8), device=DEV)
    X[:, :NFEAT] = torch.randn((rows, NFEAT), generator=gen, device=DEV)
    T = torch.stack([torch.tanh(X[:, 0] + 0.5 * X[:, 3]), 0.3 * X[:, 1] * X[:, 4]], 1).contiguous()
    order = torch.randperm(rows, generator=gen, device=DEV)
    params = torch.from_numpy(init_params(seed)).to(DEV)
    v = 1e-4 * (0.5 + torch.rand(NPARAM, generator=gen, device=DEV))
    return X, T, order, params, v


def _prepare_train(case, seed) -> dict:
    X, T, order, params, v = _train_inputs(case, seed)
    ctx, stream = api.Context(0), torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)      # the batches' gathers and the library's kernels on one stream
    return dict(case, ctx=ctx, stream=stream, X=X, T=T, order=order, params=params, m=torch.zeros_like(params), v=v,
                grad=torch.zeros(NPARAM + 1, device=DEV), step=200, at=0)


# ---- one pass ----------------------------------------------------------------
def _read_state(s) -> dict:
    L, ctx, o = api.lib(), s["ctx"], s["out"]
    at = lambda a: a.ctypes.data      # noqa: E731
    ctx._check(L.psg_get_state(ctx.h, at(o["lambdaH"]), at(o["ie"]), at(o["hits"]), at(o["lasthit"])), "psg_get_state")
    if "he" in s:
        h = s["he"]
        ctx._check(L.psg_get_he_state(ctx.h, at(h["lambdaHeI"]), at(h["lambdaHeII"]), None, None, None),
                   "psg_get_he_state")
        return dict(o, **h)
    return dict(o)


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "ticks":
        T, hits = s["ticks"], 0
        for _ in range(s["calls"]):
            if s["emit"]:
                st = ctx.run_ticks_emit(s["rays"], T, s["tick"], s["tick_time"])
            else:
                rays = s["rays"][(s["tick"] - 1) // T % HOST_BATCHES]
                st = ctx.run_ticks(rays, len(rays) // T, T, s["tick"], s["tick_time"])
            s["tick"] += T
            hits += int(st["hits"])
        return dict(_read_state(s), total_hits=hits, lost_photons=st["lost_photons"])
    if kind == "trace":
        s["tick"] += 1
        return _trace(s, s["rays"][s["tick"] % HOST_BATCHES])
    if kind == "epoch":
        ctx.load(s["field"])
        ctx.build_tree(8)
        return dict(_trace(s, s["rays"][0]), **ctx.tree_info())
    if kind == "steps":
        r = ctx.step_evolve(s["records"].copy())
        return {"lambdaH": r["lambdaH"], "ie": r["ie"]}
    with torch.cuda.stream(s["stream"]):
        return _train(s)


def _trace(s, rays):
    ctx, x = s["ctx"], s["list"]
    off = np.zeros(len(rays) + 1, np.int64)
    ctx._check(api.lib().psg_trace(ctx.h, rays.ctypes.data, len(rays), off.ctypes.data, C.byref(x.x), C.byref(x.size)),
               "psg_trace")
    hits = x.array()
    return {"off": off, "ipar": hits["ipar"], "d": hits["d"], "b": hits["b"]}


def _train(s):
    """surrogate.fit()'s inner loop."""
    L, ctx, b = api.lib(), s["ctx"], s["batch"]
    P = lambda t: C.c_void_p(t.data_ptr())      # noqa: E731
    for _ in range(s["steps"]):
        idx = s["order"][s["at"] * b:(s["at"] + 1) * b]
        s["at"] = (s["at"] + 1) % 16
        x, t = s["X"][idx].contiguous(), s["T"][idx].contiguous()
        ctx._check(L.psg_mlp_grad(ctx.h, P(s["params"]), P(x), P(t), b, P(s["grad"]), None), "psg_mlp_grad")
        s["step"] += 1
        ctx._check(L.psg_mlp_adam(ctx.h, P(s["params"]), P(s["grad"]), P(s["m"]), P(s["v"]), C.c_float(1e-3),
                                  C.c_float(0.9), C.c_float(0.999), C.c_float(1e-8), s["step"]), "psg_mlp_adam")
    return {"params": s["params"], "grad": s["grad"], "m": s["m"], "v": s["v"]}


# ---- what a pass cannot do without ---------------------------------------------
def _hits_per_ray(side, sigma):
    """Mean hits of a ray: a chord through the box times the kernels'
    cross-section, so proportional to the particles per side (measured:
    137 at 64^3 with the corner source, whose rays mostly leave the box, 785
    at 128^3 with sources inside)."""
    return (2.1 if sigma == 0.0 else 6.1 if sigma < 1.5 else 4.8) * side


def work(case) -> dict:
    """Per hit: the particle's position and smoothing length (16 bytes), its
    neutral fraction and mass (12), the absorbed photons (8, and 8 of heat
    or 24 with helium). Per updated particle and tick its state read and
    written (about 100 bytes); the state read back, 24 bytes a particle."""
    kind = case["kind"]
    if kind == "steps":
        rec = api.STEP_DTYPE.itemsize
        return {"bytes": 2 * rec * case["n"], "flops": (700 if not case["iso"] else 100) * case["n"]}
    if kind == "train":
        mlp = 2 * (8 * 64 + 64 * 64 + 2 * 64)
        return {"bytes": case["steps"] * (case["batch"] * 40 + 6 * 4 * NPARAM),
                "flops": case["steps"] * 3 * mlp * case["batch"]}
    n = case["side"] ** 3
    hits = case["rays"] * _hits_per_ray(case["side"], case["sigma"])
    if kind == "trace":
        return {"bytes": hits * (16 + 24), "flops": 40 * hits}
    if kind == "epoch":
        return {"bytes": n * (40 + 40) + hits * (16 + 24), "flops": 60 * n}
    hits *= case["ticks"] * case["calls"]
    active = min(hits / 3, n * case["ticks"] * case["calls"])
    per_hit = 36 + (24 if case["helium"] else 0 if case["iso"] else 8)
    return {"bytes": hits * per_hit + active * 100 + n * (24 + (16 if case["helium"] else 0)),
            "flops": hits * 60 + active * (100 if case["iso"] else 700)}


# ---- 64-bit values -------------------------------------------------------------
def exact(case, seed):
    """The steps' end states and the training's weights in 64 bits. The
    ticks, hit lists and trees have none: which particles a ray hits is
    decided by single-precision comparisons down the octree, and the rays'
    directions by the library's own random streams."""
    if case["kind"] == "steps":
        return _exact_steps(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed)
    return None


def _rate_columns(units):
    """The rate file's columns in internal units, with Cen's (1992)
    bremsstrahlung as the reference evaluates it (on the table's first
    column, log T)."""
    with open(api.RATES_HUI) as f:
        lines = f.read().splitlines()
    names = lines[1].replace("Log T", "logT").split()
    rows = int(lines[0].split()[2])
    data = np.array([[float(v) for v in ln.split()] for ln in lines[3:3 + rows]])
    cm3s = units.CM ** 3 / units.SEC
    col = lambda name: data[:, names.index(name)]      # noqa: E731
    return data[:, 0], {"ci": col("HIci") * cm3s, "rcB": col("HIIrcB") * cm3s,
                        "rccB": col("HIIrccB") * cm3s * units.ERG, "cic": col("HIcic") * cm3s * units.ERG,
                        "cec": col("HIcec") * cm3s * units.ERG,
                        "brem": 1.42e-27 * 1.5 * np.sqrt(data[:, 0]) * cm3s * units.ERG}


def _exact_steps(case, seed):
    """Hydrogen on the spot, solve.c:76-141, over the normalised step: 4th
    order Runge-Kutta, 2048 equal steps (isothermal with T fixed)."""
    units = Units(hmf=1.0)
    r = _step_records(case, units, seed)
    to = lambda a: torch.from_numpy(np.array(a, np.float64)).to(DEV)      # noqa: E731
    lam, ie, g, heat, time, nH, T0 = (to(r[k]) for k in ("lambdaH", "ie", "yGdepHI", "heat", "time", "nH", "T"))
    logT, cols = _rate_columns(units)
    logT0, step = float(logT[0]), float(logT[1] - logT[0])
    tab = {k: to(v) for k, v in cols.items()}

    def f(x, e):
        ye = 1.0 - x
        T = T0 if case["iso"] else units.MPROTON_OVER_BOLTZMANN * e / (1.0 + ye) * 2.0 / 3.0
        u = ((torch.log10(T) - logT0) / step).clamp(0.0, len(logT) - 1.0)
        i = u.long().clamp_max(len(logT) - 2)
        w = u - i
        at = lambda k: tab[k][i] + w * (tab[k][i + 1] - tab[k][i])      # noqa: E731
        dx = -g + time * nH * ye * (at("rcB") * ye - at("ci") * x)
        if case["iso"]:
            return dx, torch.zeros_like(e)
        loss = nH * ((at("cic") + at("cec")) * x + (at("rccB") + at("brem")) * ye)
        return dx, heat - units.H_PER_MASS * time * ye * loss

    n = 2048
    h = 1.0 / n
    for _ in range(n):
        a = f(lam, ie)
        b = f(lam + h / 2 * a[0], ie + h / 2 * a[1])
        c = f(lam + h / 2 * b[0], ie + h / 2 * b[1])
        d = f(lam + h * c[0], ie + h * c[1])
        lam = lam + h / 6 * (a[0] + 2 * b[0] + 2 * c[0] + d[0])
        ie = ie + h / 6 * (a[1] + 2 * b[1] + 2 * c[1] + d[1])
    return {"lambdaH": lam.clamp(0.0, 1.0), "ie": None if case["iso"] else ie}


def _exact_train(case, seed):
    X, T, order, params, v = _train_inputs(case, seed)
    p, v, m, b = params.double(), v.double(), torch.zeros(NPARAM, device=DEV, dtype=torch.float64), case["batch"]
    for k in range(case["steps"]):
        idx = order[k * b:(k + 1) * b]
        x, t = X[idx].double(), T[idx].double()
        q = p.detach().requires_grad_(True)
        W1, b1, W2, b2, W3, b3 = torch.split(q, [512, 64, 4096, 64, 128, 2])
        h1 = torch.nn.functional.silu(x @ W1.view(64, 8).T + b1)
        h2 = torch.nn.functional.silu(h1 @ W2.view(64, 64).T + b2)
        sse = ((h2 @ W3.view(2, 64).T + b3 - t) ** 2).sum()
        grad = torch.autograd.grad(sse / b, q)[0]
        n = 201 + k
        m = 0.9 * m + 0.1 * grad
        v = 0.999 * v + 0.001 * grad * grad
        p = p - 1e-3 * (m / (1 - 0.9 ** n)) / ((v / (1 - 0.999 ** n)).sqrt() + 1e-8)
    return {"params": p, "grad": torch.cat([grad, sse.detach()[None]]), "m": m, "v": v}
