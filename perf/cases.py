"""Performance cases of the erosion library: what a program that bakes worlds
has it do, through the public entry points of ``pgerosion``.

A case is a dict of plain values.  ``listed()`` gives the fixed ones,
``draw(rng)`` another of the same ranges, ``prepare`` builds the state a
program holds before the call (a seeded synthetic world, evolved a little so
that it has rivers, sediment and stockpiles), ``run`` makes one pass and
returns the state it leaves, ``work`` counts the bytes and operations the pass
cannot do without, and ``exact`` recomputes the map passes in plain float64
torch.

Kinds:

* ``step``: one whole erosion iteration (``maps.step``) -- spawns, the droplet
  pass, mass wasting, uplift, datum, halos.  Every pass starts from the same
  terrain (``adjoint.restore``), with the iteration's rain drawn ahead and
  resident on the device, as ``maps.SpawnFeeder`` has it.
* ``thermal``: the talus and creep passes alone.
* ``refresh``: the sea mask and the routing surface an iteration rebuilds
  every tenth time.
* ``isostasy``: the flexural response applied every twentieth iteration.
* ``calibration``: a loss of the eroded surface and its gradients.
* ``batch``: several worlds of different sizes stepped together.
"""
from __future__ import annotations

import copy
import math
import os
import sys

# 32 hardware queues for the batched worlds, as the benchmark sets them (read when CUDA starts)
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

import numpy as np
import torch

PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "procedural-generation_b200")
if PACKAGE not in sys.path:
    sys.path.insert(0, PACKAGE)

from pgerosion import _lib, adjoint, batch, isostasy  # noqa: E402
from pgerosion import maps  # noqa: E402
from pgerosion.geometry import BASES, get_grid  # noqa: E402
from pgerosion.params import ErosionParams, WorldGroup, WorldParams, cell_units, plain_knobs  # noqa: E402
from pgerosion.synth import fbm  # noqa: E402

EARTH_CELL_M = 9773.0 * 1024.0  # the Earth-default planet: cell size times cells per face edge
HALO = 2


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # the smallest world the repository's tests step (a preview, a unit test): 16 short waves, all latency
        dict(name="tiny_step", kind="step", N=32, droplets=4096, life=64, apply="ordered", knobs="plain", brush=0, lateral=0.0),
        # the small preset: N_c = 128, 65,536 droplets, lifetime 64, faster rates
        dict(name="small_step", kind="step", N=128, droplets=65536, life=64, apply="ordered", knobs="small", brush=0, lateral=0.0),
        # the headline: the Earth-default world, 1,572,864 droplets, lifetime 96, the exact apply
        dict(name="earth_step", kind="step", N=1024, droplets=1572864, life=96, apply="ordered", knobs="plain", brush=0, lateral=0.0),
        # the bake's default knobs (routing surface, lakes with their parks, isostatic load) and lifetime 2 N
        dict(name="lakes_step", kind="step", N=256, droplets=98304, life=0, apply="ordered", knobs="bake", brush=0, lateral=0.0),
        # a zoom tile: one masked face of odd size, roots and the bank cut on, droplets leave over its edge
        dict(name="window_step", kind="step", N=389, droplets=37831, life=160, apply="ordered", knobs="window", brush=0, lateral=0.5),
        # the order-free apply on the Earth-default world, one wave an iteration
        dict(name="wave_step", kind="step", N=1024, droplets=1572864, life=96, apply="wave", knobs="plain", brush=0, lateral=0.0),
        # the planet level's options (brush of radius 2, lifetime 128) on a ragged size
        dict(name="brush_step", kind="step", N=601, droplets=90301, life=128, apply="wave", knobs="plain", brush=2, lateral=0.0),
        # mass wasting alone, N_c = 1024
        dict(name="thermal", kind="thermal", N=1024),
        # the sea mask and routing surface of an evolved world, N_c = 1024
        dict(name="refresh", kind="refresh", N=1024),
        # the isostatic response, odd size
        dict(name="isostasy", kind="isostasy", N=725),
        # the calibration's loss and gradients, forward and backward
        dict(name="calibration", kind="calibration", N=96, droplets=18432, iterations=4, every=2),
        # uneven worlds stepped at once on one GPU
        dict(name="batch", kind="batch", worlds=10, largest=256, mix=10),
    ]


def _size(rng, lo, hi):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(lo, min(hi, n + rng.choice((0, 0, 1))))


def draw(rng):
    kind = rng.choice(("step",) * 7 + ("thermal", "refresh", "isostasy", "calibration", "batch"))
    if kind in ("thermal", "refresh", "isostasy"):
        return dict(kind=kind, N=_size(rng, 96, 725) if kind == "isostasy" else _size(rng, 32, 1024))
    if kind == "calibration":
        N = _size(rng, 32, 96)
        return dict(kind=kind, N=N, droplets=max(256, int(2 * N * N * rng.uniform(0.4, 1.0))), iterations=rng.choice((2, 3, 4)), every=2)
    if kind == "batch":
        return dict(kind=kind, worlds=rng.randint(3, 10), largest=rng.choice((128, 192, 256)), mix=rng.randrange(1 << 16))
    what = rng.choice(("plain", "plain", "small", "bake", "window", "wave", "wave"))
    N = _size(rng, 32, {"plain": 1024, "small": 256, "bake": 256, "window": 389, "wave": 1024}[what])
    cells = N * N * (1 if what == "window" else 6)
    lo, hi = {"small": (0.25, 0.6)}.get(what, (0.05, 0.25))
    c = dict(kind="step", N=N, droplets=max(33, int(cells * rng.uniform(lo, hi))), life=rng.choice((64, 96, 128)), apply="ordered",
             knobs="plain" if what == "wave" else what, brush=0, lateral=0.0)
    if what == "plain" and c["life"] == 128:
        c["life"] = 96
    if what == "bake":
        c["life"] = rng.choice((0, 96))
    elif what == "window":
        c["life"], c["lateral"] = rng.choice((96, 160)), rng.choice((0.0, 0.5))
    elif what == "wave":
        c["apply"], c["brush"] = "wave", rng.choice((0, 0, 2, 3))
        c["life"] = 96
    return c


# --------------------------------------------------------------------------
# seeded worlds, built on the device
# --------------------------------------------------------------------------
def _points(N, faces, dev):
    """(faces, N, N, 3) unit vectors of the interior cell centres (the equi-angular cube-sphere)."""
    e = (torch.arange(N, dtype=torch.float64, device=dev) + 0.5) / N
    t = torch.tan((e - 0.5) * (math.pi / 2.0))
    s, u = torch.meshgrid(t, t, indexing="ij")
    B = torch.as_tensor(BASES, device=dev)[:faces]
    q = B[:, 2, None, None, :] + s[None, ..., None] * B[:, 0, None, None, :] + u[None, ..., None] * B[:, 1, None, None, :]
    return q / q.norm(dim=-1, keepdim=True)


def _world(N, seed, cell, land=0.29, window=False, lo=-8000.0, hi=6000.0):
    """An Earth-like ErosionState: fBm plus ridges rank-mapped to lo..hi metres with ``land`` of it above
    the sea, latitude-banded rain 0.1..3, uplift 0..2 mm an iteration, hardness 0.5 +- 0.25."""
    dev = torch.device("cuda")
    F, NE, H = (1 if window else 6), N + 2 * HALO, HALO
    grid = get_grid(N, H, cell)
    rng = np.random.default_rng([seed, N])
    p = _points(N, F, dev)
    v = fbm(p, rng, 6) + 0.6 * fbm(p, rng, 4, base_freq=4.0, ridged=True)
    s = torch.sort(v.reshape(-1)).values
    q, v0, v1 = s[int((1.0 - land) * (s.numel() - 1))], s[0], s[-1]
    bed = torch.where(v < q, lo * (q - v) / (q - v0), hi * (v - q) / (v1 - q)) / cell
    lat = torch.asin(p[..., 2].clamp(-1.0, 1.0))
    band = torch.exp(-(lat / 0.25) ** 2) + 0.6 * torch.exp(-((lat.abs() - 1.0) / 0.2) ** 2)
    rain = (0.1 + 2.9 * band / band.max() * (0.6 + 0.8 * (0.5 + 0.5 * fbm(p, rng, 4)))).clamp(0.1, 3.0)
    upl = 0.002 / cell * (0.5 + 0.5 * fbm(p, rng, 4)).clamp(0.0, 1.0)
    hard = (0.5 + 0.25 * fbm(p, rng, 4)).clamp(0.0, 1.0)

    def field(x=None, pad=0.0):
        f = torch.full((F, NE, NE), pad, dtype=torch.float64, device=dev)
        if x is not None:
            f[:, H:H + N, H:H + N] = x
        return f

    mask = None
    if window:  # a round basin of active cells, a frozen margin around it, nothing in the corners
        i = (torch.arange(NE, dtype=torch.float64, device=dev) - 0.5 * (NE - 1)) / (0.5 * N)
        r = torch.sqrt(i[:, None] ** 2 + i[None, :] ** 2)[None]
        mask = torch.where(r < 0.98, 1, torch.where(r < 1.25, 2, 0)).to(torch.uint8)
        mask[:, :H] = mask[:, -H:] = 0
        mask[:, :, :H] = mask[:, :, -H:] = 0
    st = maps.ErosionState(
        height=field(bed), sediment=field(), discharge=field(), momentum=torch.zeros((F, NE, NE, 2), dtype=torch.float64, device=dev),
        hardness=field(hard, 0.5).float(), precip=field(rain, 0.1).float(), evap=field(pad=1.0).float(), uplift=field(upl), mask=mask,
        metric=torch.as_tensor(np.ascontiguousarray(grid.metric_face), device=dev),
        metric_inv=torch.as_tensor(np.ascontiguousarray(grid.metric_inv_face), device=dev), N=N, H=H, spherical=not window,
        height_unit_m=float(cell), grid=grid, land_target=land, deposit_on_exit=window)
    st.exchange_halos()
    return st


def _params(case, seed):
    N, life = case["N"], case["life"]
    if case["knobs"] == "small":
        ep = ErosionParams(iterations=20, max_steps=life, friction=0.05, erodibility=0.3, deposition_rate=0.3, evap_rate=0.01,
                           uplift_mode="stack", **plain_knobs())
        return WorldParams(world=WorldGroup(seed=seed, N_c=N, cell_size_m=50.0, land_fraction=0.30, halo=HALO), erosion=ep)
    if case["knobs"] == "bake":
        ep = ErosionParams(max_steps=life, ice_sheet=False)
    elif case["knobs"] == "window":
        ep = ErosionParams(iterations=80, max_steps=life, uplift_mode="stack", disc_saturation_cells=32.0, momentum_saturation_cells=1.0,
                           **dict(plain_knobs(), lateral_rate=case["lateral"]))
    else:
        ep = ErosionParams(iterations=400, max_steps=life, uplift_mode="replay", brush_radius=case["brush"], **plain_knobs())
    cell = 300.0 if case["knobs"] == "window" else EARTH_CELL_M / N
    return WorldParams(world=WorldGroup(seed=seed, N_c=N, cell_size_m=cell, land_fraction=0.29, halo=HALO), erosion=ep)


def _rain(params, key, P):
    """One iteration's rain draws on the device and the generator that follows them (maps.SpawnFeeder)."""
    rng, u, off = maps.draw_spawns(params, "erosion", (key,), P)
    return rng, torch.as_tensor(u, device="cuda"), torch.as_tensor(off, device="cuda")


def _evolve(st, params, P, iterations=2):
    """A few order-free iterations: rivers, sediment and stockpiles before the measured pass."""
    p = params.with_erosion(brush_radius=0, flood_every=0, sea_mask_every=0, lake_balance=False, lake_fill=False, glacial_every=0,
                            isostasy=0.0)
    for k in range(iterations):
        maps.step(st, p, 900 + k, n_particles=P, apply=_lib.APPLY_WAVE, wave=2 * P + 4096)


def _evolved(N, seed, cell=None):
    c = dict(N=N, life=96, knobs="plain", brush=0)
    p = _params(c, seed)
    st = _world(N, seed, EARTH_CELL_M / N if cell is None else cell)
    _evolve(st, p, max(64, 6 * N * N // 8))
    return st, p


# --------------------------------------------------------------------------
# prepare / run
# --------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        return _prepare_step(case, seed)
    if kind == "batch":
        return _prepare_batch(case, seed)
    if kind == "calibration":
        return _prepare_calibration(case, seed)
    st, p = _evolved(case["N"], seed)
    s = dict(kind=kind, st=st, params=p, snap=adjoint.snapshot(st))
    if kind == "isostasy":
        s["params"] = p.with_erosion(isostasy=0.8, flexure_km=60.0)
        s["acc"] = _load(st, seed)
        st.iso_acc = s["acc"].clone()
        isostasy.smoothing_kappa(st)  # the grid's step bound, found once
    if kind == "refresh":
        st.owner_table()
    return s


def _load(st, seed):
    """What twenty iterations took from and put on each cell: a seeded field of some metres."""
    dev = st.height.device
    f = torch.zeros_like(st.height)
    g = torch.Generator(device=dev).manual_seed(seed)
    f[st.interior] = torch.randn((st.F, st.N, st.N), dtype=torch.float64, device=dev, generator=g) * (20.0 / st.height_unit_m)
    return f


def _prepare_step(case, seed):
    params = _params(case, seed)
    ep = params.erosion
    window = case["knobs"] == "window"
    lo, hi = {"small": (-4000.0, 3000.0), "window": (-400.0, 2500.0)}.get(case["knobs"], (-8000.0, 6000.0))
    land = 0.85 if window else params.world.land_fraction
    st = _world(case["N"], seed, params.world.cell_size_m, land=land, window=window, lo=lo, hi=hi)
    maps.start_replay(st, params)
    P = case["droplets"]
    if window:
        st.roots = (0.5 * st.hardness).contiguous()
        st.inflow_volume = 0.05 * P
    _evolve(st, params, P)
    if case["knobs"] == "bake":
        # what the last refresh (every tenth iteration) left: base level, routing surface, lakes with room
        st.refresh_base(maps.ocean_min_fraction(params))
        st.refresh_route(cell_units(ep, "route_eps", st.height_unit_m))
        st.refresh_lakes(params.hydro.lake_evap, maps.lake_min_depth(params) / st.height_unit_m, params.hydro.ocean_min_fraction,
                         params.hydro.land_evap, fill=maps.lake_fill_args(st, params))
        st.ensure_lake_parks()
        st.iso_acc = torch.zeros_like(st.height)
    st.iteration = 3
    kw = dict(n_particles=P)
    if case["apply"] == "wave":
        kw.update(apply=_lib.APPLY_WAVE, wave=2 * P + 4096)
    more = {k: getattr(st, k).clone() for k in ("route", "lake_load", "lake_room", "iso_acc") if getattr(st, k) is not None}
    return dict(kind="step", st=st, params=params, snap=adjoint.snapshot(st), more=more, rain=_rain(params, 3, P), kw=kw)


def _prepare_batch(case, seed):
    sizes = [n for n in batch.BATCH_SIZES if n <= case["largest"]]
    worlds = batch.batch_worlds(case["worlds"], seed=case["mix"], sizes=sizes)
    states, params, counts, rain = [], [], [], []
    for w in worlds:
        w.params.world.seed = seed + len(states)
        st = _world(w.N, w.params.world.seed, w.params.world.cell_size_m)
        maps.start_replay(st, w.params)
        _evolve(st, w.params, w.n_particles, 1)
        st.iteration = 3
        states.append(st)
        params.append(w.params)
        counts.append(w.n_particles)
        rain.append(_rain(w.params, 3, w.n_particles))
    runner = batch.Runner(states, params, costs=[w.cost for w in worlds])
    return dict(kind="batch", runner=runner, states=states, counts=counts, rain=rain, snaps=[adjoint.snapshot(s) for s in states])


def _prepare_calibration(case, seed):
    N = case["N"]
    p = adjoint.calibration_params(seed=seed, N=N, iterations=case["iterations"])
    st = _world(N, seed, p.world.cell_size_m)
    maps.start_replay(st, p)
    calib = adjoint.Calibration(st, p, case["iterations"], case["droplets"], checkpoint_every=case["every"])
    target = calib.run(None, adjoint.rates_of(adjoint.calibration_params(seed=seed, N=N, jitter=0.3)).tolist())
    land = torch.zeros_like(target, dtype=torch.bool)
    land[st.interior] = target[st.interior] > 0.0
    return dict(kind="calibration", calib=calib, target=target, land=land, unit=st.height_unit_m,
                erod=adjoint.erodibility_init(st, seed), rates=adjoint.rates_of(p).to(st.height.device))


def _fields(st):
    return {k: getattr(st, k) for k in adjoint.PASS_FIELDS}


def run(s):
    kind = s["kind"]
    if kind == "step":
        st = s["st"]
        adjoint.restore(st, s["snap"])
        for k, v in s["more"].items():
            getattr(st, k).copy_(v)
        rng, u, off = s["rain"]
        stats = maps.step(st, s["params"], st.iteration, predrawn=(copy.deepcopy(rng), u, off), **s["kw"])
        # (the lakes' rooms are one value a lake, another number of them on every world)
        out = _fields(st) | {k: getattr(st, k) for k in s["more"] if k != "lake_room"}
        out["droplet_steps"] = stats["droplet_steps"]
        return out
    if kind == "batch":
        for st, snap in zip(s["states"], s["snaps"]):
            adjoint.restore(st, snap)
        rain = s["rain"]
        s["runner"].step(1, n_particles=s["counts"], spawns=lambda i, it: (copy.deepcopy(rain[i][0]), rain[i][1], rain[i][2]))
        return [(st.height, st.sediment, st.discharge, st.momentum, st.pending) for st in s["states"]]
    if kind == "calibration":
        erod = s["erod"].clone().requires_grad_(True)
        rates = s["rates"].clone().requires_grad_(True)
        z = adjoint.erode(erod, rates, s["calib"])
        loss = adjoint.land_loss(z, s["target"], s["land"], s["unit"])
        loss.backward()
        return z.detach(), loss.detach(), erod.grad, rates.grad
    st = s["st"]
    if kind == "thermal":
        st.height.copy_(s["snap"]["height"])
        st.sediment.copy_(s["snap"]["sediment"])
        maps.thermal_erosion(st, s["params"])
        return st.height, st.sediment
    if kind == "isostasy":
        st.height.copy_(s["snap"]["height"])
        st.iso_acc.copy_(s["acc"])
        isostasy.apply_isostasy(st, s["params"])
        return st.height
    p = s["params"]
    st.refresh_base(maps.ocean_min_fraction(p))
    st.refresh_route(cell_units(p.erosion, "route_eps", st.height_unit_m))
    return st.base, st.sea_mask, st.route


# --------------------------------------------------------------------------
# work
# --------------------------------------------------------------------------
#: one droplet step: its gathers and scatters (105 B read, 32 B of sums) and float64 operations
STEP_BYTES, STEP_FLOPS = 137, 250
#: steps a droplet lives on these worlds, as a share of its lifetime up to 96 steps
MEAN_LIFE = 0.55
#: the map passes of an iteration: the state read and written once
CELL_BYTES, CELL_FLOPS = 180, 200


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes = [n for n in batch.BATCH_SIZES if n <= case["largest"]]
        one = [work(dict(kind="step", N=n, droplets=6 * n * n // 8, life=0, knobs="plain", brush=0)) for n in sizes]
        return {k: case["worlds"] * sum(w[k] for w in one) / len(one) for k in ("bytes", "flops")}
    if kind == "calibration":  # forward, recomputed forward and the reverse
        w = work(dict(kind="step", N=case["N"], droplets=case["droplets"], life=0, knobs="plain", brush=0))
        return {k: 3 * case["iterations"] * v for k, v in w.items()}
    cells = (1 if case.get("knobs") == "window" else 6) * (case["N"] + 2 * HALO) ** 2
    if kind == "step":
        life = min(case["life"] or 2 * case["N"], 96)
        steps = case["droplets"] * MEAN_LIFE * life
        per = STEP_BYTES + (8 * {2: 25, 3: 45}[case["brush"]] if case["brush"] else 0)
        return {"bytes": steps * per + cells * CELL_BYTES, "flops": steps * STEP_FLOPS + cells * CELL_FLOPS}
    if kind == "thermal":  # height and sediment in and out, hardness, base
        return {"bytes": 44 * cells, "flops": 2 * 8 * 12 * cells}
    if kind == "refresh":  # height, sediment, owner in; base, route and the open sea out
        return {"bytes": 37 * cells, "flops": 16 * cells}
    # the load and the height in, the height out
    return {"bytes": 24 * cells, "flops": 60 * cells}


# --------------------------------------------------------------------------
# the map passes in plain float64
# --------------------------------------------------------------------------
D8 = ((1, 0), (1, 1), (0, 1), (-1, 1), (-1, 0), (-1, -1), (0, -1), (1, -1))


def exact(case, seed):
    if case["kind"] == "thermal":
        return _exact_thermal(prepare(case, seed))
    if case["kind"] == "refresh":
        return _exact_refresh(prepare(case, seed))
    if case["kind"] == "isostasy":
        return _exact_isostasy(prepare(case, seed))
    return None  # a droplet pass is a serial walk of every droplet: no plain form within seconds


def _exact_thermal(s):
    st, ep, unit = s["st"], s["params"].erosion, s["st"].height_unit_m
    h, d = st.height.clone(), st.sediment.clone()
    g = st.metric.double()
    talus = (torch.tensor(ep.talus_slope_soft, dtype=torch.float32, device=h.device)
             + torch.tensor(ep.talus_slope_hard - ep.talus_slope_soft, dtype=torch.float32, device=h.device) * st.hardness).double()
    cap, floor = cell_units(ep, "thermal_max", unit), cell_units(ep, "dep_floor_m", unit)
    roll = lambda a, k, sign=1: torch.roll(a, (-sign * D8[k][0], -sign * D8[k][1]), (1, 2))  # the neighbour's value
    inner = torch.zeros_like(h, dtype=torch.bool)
    inner[:, 1:-1, 1:-1] = True
    for creep, rate in ((False, ep.thermal_rate), (True, ep.creep_rate)):
        z = h + d
        active = ~(z < st.base) if creep else torch.ones_like(inner)
        flow = []
        for k, (di, dj) in enumerate(D8):
            dist = torch.sqrt(g[..., 0] * di * di + 2.0 * g[..., 1] * di * dj + g[..., 2] * dj * dj)
            drop = z - roll(z, k)
            over = drop - (0.0 if creep else talus) * dist
            flow.append(torch.where((drop > 0) & (over > 0), 0.5 * rate * over, torch.zeros_like(z)))
        sent = [torch.where(roll(active, k), f, torch.zeros_like(f)) for k, f in enumerate(flow)]
        S, mx = sum(sent), torch.stack(sent).amax(0)
        sc = torch.where(S > 2.0 * mx, 2.0 * mx / S.clamp_min(1e-300), torch.ones_like(S))
        sc = torch.where(S * sc > cap, cap / S.clamp_min(1e-300), sc)
        sc = torch.where(inner & active & (S > 0), sc, torch.zeros_like(S))
        came = [roll(sc * flow[(k + 4) % 8], k) for k in range(8)]
        inflow = sum(came)
        room = (-floor - z).clamp_min(0.0)
        rs = torch.where(inner & active & (z < 0) & (inflow > room), room / inflow.clamp_min(1e-300), torch.ones_like(z))
        out = sum(sc * roll(rs, k) * sent[k] for k in range(8))
        take, out = inner & active, torch.where(inner & active, out, torch.zeros_like(z))
        dig = (out > 0) & (d < out)  # (a halo's sediment may be below zero: interpolated)
        h = torch.where(dig, h - (out - d), h)
        d = torch.where(dig, torch.zeros_like(d), d - out) + torch.where(take, inflow * rs, torch.zeros_like(z))
    return h, d


def _neighbours(st, owner):
    """(8, cells) flat interior cell that owns each neighbour of each interior cell."""
    N, H, NE = st.N, st.H, st.NE
    return torch.stack([owner[:, H + a:H + a + N, H + b:H + b + N].reshape(-1) for a, b in D8])


def _exact_refresh(s):
    st, p = s["st"], s["params"]
    N, H, NE = st.N, st.H, st.NE
    dev = st.height.device
    owner = torch.as_tensor(np.ascontiguousarray(st.grid.owner), device=dev)
    z = (st.height + st.sediment).reshape(-1)
    inner = torch.zeros((6, NE, NE), dtype=torch.bool, device=dev)
    inner[:, H:H + N, H:H + N] = True
    cells = torch.nonzero(inner.reshape(-1))[:, 0]
    nb = _neighbours(st, owner)
    # bodies of water below the datum, joined over the eight neighbours
    big = z.numel()
    below = torch.zeros(big, dtype=torch.bool, device=dev)
    below[cells] = z[cells].float() < 0
    label = torch.where(below, torch.arange(big, device=dev), torch.full_like(owner.reshape(-1), big))
    label = torch.cat([label, torch.tensor([big], device=dev)])
    while True:
        m = torch.minimum(label[cells], label[nb].amin(0))
        new = label.clone()
        new[cells] = torch.where(below[cells], m, label[cells])
        old = label[cells]
        new.scatter_reduce_(0, torch.where(below[cells], old, big), torch.where(below[cells], m, big), "amin")
        new = new[new]
        if torch.equal(new, label):
            break
        label = new
    lab = label[cells]
    g = st.metric[H:H + N, H:H + N].double()
    area = (torch.sqrt(g[..., 0] * g[..., 2] - g[..., 1] ** 2) * st.grid.cell_size_m ** 2).expand(6, N, N).reshape(-1)
    size = torch.zeros(big + 1, dtype=torch.float64, device=dev).index_add_(0, lab, area)
    size[big] = 0.0
    floor = torch.zeros(big + 1, dtype=torch.float64, device=dev).scatter_reduce_(0, lab, z[cells], "amin")
    water = below[cells]
    open_sea = water & ((size[lab] >= maps.ocean_min_fraction(p) * area.sum()) | (lab == size.argmax()))
    base = torch.zeros_like(z)
    base[cells] = torch.where(water & ~open_sea, floor[lab], torch.zeros_like(floor[lab]))
    hm = st.grid.halo
    dst, near = (torch.as_tensor(np.ascontiguousarray(a), device=dev) for a in (hm.dst, hm.nearest))
    base[dst] = base[near]
    # the surface a flood from the sea fills, each cell at least eps above the one it came from
    eps = cell_units(p.erosion, "route_eps", st.height_unit_m)
    seed = (z[cells] < 0) & (z[cells] <= base[cells])
    r = torch.full_like(z, math.inf)
    r[cells] = torch.where(seed, z[cells], r[cells])
    while True:
        best = torch.where(seed, r[cells], torch.maximum(z[cells], r[nb].amin(0) + eps))
        if torch.equal(best, r[cells]):
            break
        r[cells] = best
    r = torch.where(torch.isinf(r), z, r)
    w, src = torch.as_tensor(np.ascontiguousarray(hm.w_lin), device=dev), torch.as_tensor(np.ascontiguousarray(hm.src), device=dev)
    r[dst] = (w * r[src]).sum(1)
    return base.reshape(6, NE, NE), None, r.reshape(6, NE, NE)


def _exact_isostasy(s):
    st, ep = s["st"], s["params"].erosion
    N, H, NE = st.N, st.H, st.NE
    dev = st.height.device
    hm = st.grid.halo
    dst, src, w, wl = (torch.as_tensor(np.ascontiguousarray(a), device=dev) for a in (hm.dst, hm.src, hm.w, hm.w_lin))
    G = torch.as_tensor(np.ascontiguousarray(st.grid.metric_inv_face), device=dev).double()
    m = torch.as_tensor(np.ascontiguousarray(st.grid.metric_face), device=dev).double()
    sq = torch.sqrt(m[..., 0] * m[..., 2] - m[..., 1] ** 2)

    def fill(f, weights):
        v = f.reshape(-1)
        v[dst] = (weights * v[src]).sum(1)

    def lap(f):
        c = lambda a, i, j: a[..., 1 + i:NE - 1 + i, 1 + j:NE - 1 + j]
        D = lambda i, j: c(f, i, j)
        Sq = lambda i, j: c(sq, i, j)
        Gk = lambda k, i, j: c(G[..., k], i, j)
        dj = lambda i: 0.5 * (D(i, 1) - D(i, -1))
        di = lambda j: 0.5 * (D(1, j) - D(-1, j))
        mid = lambda a, b: 0.5 * (a + b)

        def flux_i(a):  # between the cell and its neighbour a cells along i
            lo, hi = (0, 1) if a > 0 else (-1, 0)
            return mid(Sq(0, 0), Sq(a, 0)) * (mid(Gk(0, 0, 0), Gk(0, a, 0)) * (D(hi, 0) - D(lo, 0)) +
                                              mid(Gk(1, 0, 0), Gk(1, a, 0)) * 0.5 * (dj(0) + dj(a)))

        def flux_j(a):
            lo, hi = (0, 1) if a > 0 else (-1, 0)
            return mid(Sq(0, 0), Sq(0, a)) * (mid(Gk(2, 0, 0), Gk(2, 0, a)) * (D(0, hi) - D(0, lo)) +
                                              mid(Gk(1, 0, 0), Gk(1, 0, a)) * 0.5 * (di(0) + di(a)))

        out = torch.zeros_like(f)
        out[:, 1:-1, 1:-1] = (flux_i(1) - flux_i(-1) + flux_j(1) - flux_j(-1)) / Sq(0, 0)
        return out

    # the largest monotone step: 0.9 over the operator's largest eigenvalue, by power iteration
    f = torch.zeros((6, NE, NE), dtype=torch.float64, device=dev)
    f[st.interior] = torch.as_tensor(np.random.default_rng(0).standard_normal((6, N, N)), device=dev)
    fill(f, w)
    for _ in range(40):
        fill(f, wl)
        v = lap(f)
        num, lam = v[st.interior].norm(), v[st.interior].norm() / f[st.interior].norm()
        f = v / num
    kappa = 0.9 / float(lam)
    sig = min(ep.flexure_km * 1000.0 / st.height_unit_m, N / 8.0)
    f = -ep.isostasy * s["acc"]
    for _ in range(int(math.ceil(sig * sig / (2.0 * kappa))) if sig >= 0.5 else 0):
        fill(f, wl)
        f = f + kappa * lap(f)
    fill(f, wl)
    return s["snap"]["height"] + (f - f[st.interior].mean())
