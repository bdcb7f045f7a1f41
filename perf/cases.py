"""Timed workloads of the flood engine: the calls its users make, over the sizes, precisions
and options they use them with.

``listed()`` names the fixed cases and ``draw(rng)`` makes further ones of the same ranges.
``prepare(case, seed)`` builds what a program holds before the call (solver objects over a
state in the middle of a storm), ``run(state)`` is one pass through the public entry points,
``work(case)`` the bytes and operations a pass cannot do without, and ``exact(case, seed)``
the outputs of a pass from a plain float64 torch evaluation of the method.

Kinds of case:

* ``grid``     ``SWE2D.max_dt`` and ``SWE2D.step``: one CFL step of the 2-D model
* ``channel``  ``SWE1D.max_dt`` and ``SWE1D.substeps``: the 1-D network over one 2-D step
* ``weir``     ``exchange``: the weir links between the two models
* ``coupled``  ``CoupledEngine.step``: the host-driven coupled step
* ``resident`` ``FloodEngine.advance``: several coupled steps on the device
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch
import torch.nn.functional as F

from his_gb300 import workloads as W
from his_gb300.assembly import build_engine, build_engine_batch
from his_gb300.boundaries import EDGES, EdgeBC
from his_gb300.config import SolverConfig
from his_gb300.coupling import exchange, links_from_cells
from his_gb300.engine import FloodEngine, Member
from his_gb300.infiltration import Horton
from his_gb300.swe1d import SWE1D
from his_gb300.swe2d import SWE2D
from his_gb300.topology import build_topology, sections

KIND_OF = {"T": "transmissive", "C": "closed", "S": "stage", "D": "discharge"}
WEIR_DT = 0.002           # s: small, so that repeated passes keep moving water
RAIN = 20.0 * W.MMH       # rain of the grid cases [m/s]
SEA_LEVEL = 0.6           # stage of the grid cases' stage edges [m]
EDGE_INFLOW = 0.8         # inflow of their discharge edges [m^2/s]


def listed():
    return [
        # a small district at 80 m, plain method, stepped by the caller as the verification
        # cases do: few cells, so the length of the dependent chain and the launches count
        dict(name="grid_small_f64", kind="grid", dtype="float64", nx=100, ny=81, dx=80.0, members=1, order=2,
             flux="hllc", edges="TTST", sources=False, weights=False),
        # the full-resolution catchment, plain method, infiltration and retention on
        dict(name="grid_full_f64", kind="grid", dtype="float64", nx=400, ny=325, dx=20.0, members=1, order=2,
             flux="hllc", edges="TTST", sources=True, weights=False),
        # screening runs: first order, HLL, rain weights, walls and an inflow edge, odd sizes
        dict(name="grid_first_order_f32", kind="grid", dtype="float32", nx=163, ny=201, dx=40.0, members=3, order=1,
             flux="hll", edges="CTDT", sources=True, weights=True),
        # one large domain at 5 m in the production form
        dict(name="grid_large_f32", kind="grid", dtype="float32", nx=1601, ny=1301, dx=5.0, members=1, order=2,
             flux="hllc", edges="TTST", sources=True, weights=False),
        # the channel network alone, one storm: three reaches and a junction
        dict(name="channel_f64", kind="channel", dtype="float64", nx=400, ny=325, dx=20.0, members=1, span=5.0),
        # the weir links of a batch in the production form
        dict(name="weir_batch_f32", kind="weir", dtype="float32", nx=400, ny=325, dx=20.0, members=16),
        # the host-driven coupled step: one small storm in the plain method
        dict(name="coupled_small_f64", kind="coupled", dtype="float64", nx=100, ny=81, dx=80.0, members=1),
        # and the 64-storm batch in the production form
        dict(name="coupled_batch_f32", kind="coupled", dtype="float32", nx=400, ny=325, dx=20.0, members=64),
        # the resident loop: one full-resolution storm in the plain method
        dict(name="resident_full_f64", kind="resident", dtype="float64", grids="400x325@20*1", steps=4, tile_y=16,
             peaks=False),
        # a handful of storms of mixed sizes, as the server steps them between admissions
        dict(name="resident_served_f32", kind="resident", dtype="float32", grids="100x81@80*2,200x163@40*2,400x325@20*2",
             steps=16, tile_y=16, peaks=True),
        # the 64-storm batch of the headline metric
        dict(name="resident_batch_f32", kind="resident", dtype="float32", grids="400x325@20*64", steps=16, tile_y=64,
             peaks=False),
    ]


def draw(rng):
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    kind = rng.choice(["grid", "grid", "grid", "channel", "weir", "coupled", "coupled", "resident", "resident"])
    dtype = rng.choice(["float64", "float32"])
    f64 = dtype == "float64"
    if kind == "resident":
        most = 3 if f64 else 24
        grids, cells = [], 0
        for nx, ny, dx in rng.sample([(100, 81, 80), (200, 163, 40), (400, 325, 20)], rng.randint(1, 3)):
            nx, ny = nx - rng.randint(0, 17), ny - rng.randint(0, 17)
            k = log(1, most)
            if cells + nx * ny * k > (200_000 if f64 else 4_000_000):
                k = 1
            cells += nx * ny * k
            grids.append(f"{nx}x{ny}@{dx}*{k}")
        return dict(kind=kind, dtype=dtype, grids=",".join(grids), steps=4 if f64 else 16,
                    tile_y=rng.choice([16, 24, 32, 48, 64]), peaks=rng.random() < 0.5)
    dx = float(rng.choice([10, 20, 40, 80]))
    if kind == "grid":
        nx, ny = log(60, 420 if f64 else 1400), log(60, 340 if f64 else 1200)
        members = max(1, min(log(1, 24), (200_000 if f64 else 3_000_000) // (nx * ny)))
        return dict(kind=kind, dtype=dtype, nx=nx, ny=ny, dx=dx, members=members, order=rng.choice([1, 2, 2, 2]),
                    flux=rng.choice(["hllc", "hllc", "hll"]), edges="".join(rng.choice("TTCSD") for _ in range(4)),
                    sources=rng.random() < 0.6, weights=rng.random() < 0.3)
    nx, ny = log(90, 420), log(81, 340)
    members = max(1, min(log(1, 64), (150_000 if f64 and kind == "coupled" else 3_000_000) // (nx * ny)))
    case = dict(kind=kind, dtype="float64" if kind == "channel" else dtype, nx=nx, ny=ny, dx=max(dx, 20.0), members=members)
    return dict(case, span=rng.choice([1.0, 5.0, 20.0])) if kind == "channel" else case


# ------------------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=16)
def _terrain(nx, ny, dx):
    """The seeded valley terrain of the repository's workloads; small grids carry one reach,
    the others three reaches and a junction."""
    return W.make_terrain(nx, ny, float(dx), 24 if nx >= 200 else 12, f"perf/{nx}x{ny}",
                          "single" if nx * ny < 10_000 else "triple")


@functools.lru_cache(maxsize=64)
def _bank_links(nx, ny, dx):
    ter = _terrain(nx, ny, dx)
    return W.bank_links(ter, build_topology(_network(ter, 1.0)))


def _network(ter, gamma):
    return W.make_network(ter, "single" if ter.junction is None else "triple", gamma)


def _storms(nx, ny, dx, members, seed, first=0):
    """Storms of the batch workload's draws (roughness, retention, infiltration, conveyance,
    rain, tide, inflow), with the clock at zero in the middle of the rain.  They last two
    days, so that no number of passes reaches their end."""
    ter = _terrain(nx, ny, dx)
    shp, out = (ter.ny, ter.nx), []
    for b in range(first, first + members):
        r = np.random.default_rng([seed, b])
        q_peak = r.uniform(100.0, 600.0) * (0.1 if ter.junction is None else 1.0)
        f = W.Forcing(rain_t0=-3 * 3600.0, rain_step=600.0, rain=W.alternating_block(6 * 3600.0, 600.0, r.uniform(40, 80)),
                      tide_on=True, q_t0=-4 * 3600.0, q_step=60.0,
                      q=W.triangular_inflow(12 * 3600.0, q_peak, 0.05 * q_peak, 5 * 3600.0, 3 * 3600.0),
                      **W.m2_tide(r.uniform(0.5, 1.5), 1800.0))
        horton = (np.full(shp, r.uniform(30, 90) * W.MMH), np.full(shp, 8.0 * W.MMH), np.full(shp, 4.0 / 3600.0), 0.0)
        out.append(W.Storm(f"perf/{seed}/{b}", ter, r.uniform(0.02, 0.06), np.full(shp, r.uniform(0.001, 0.010)),
                           horton, f, 48 * 3600.0, _network(ter, r.uniform(0.7, 1.3))))
    return out


def _flooded(ter, members, seed, dtype, storage):
    """A state in the middle of a storm: runoff films with dry patches on the hills, water
    standing in the hollows and the channel, smooth velocities; partly filled storage."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    z = torch.as_tensor(ter.z, device="cuda")
    ny, nx = z.shape
    noise = lambda: F.interpolate(torch.rand(members, 1, 3 + ny // 24, 3 + nx // 24, generator=g, device="cuda",
                                             dtype=torch.float64), (ny, nx), mode="bilinear", align_corners=True)[:, 0]
    plain = F.avg_pool2d(F.pad(z[None, None], (7, 7, 7, 7), mode="replicate"), 15, 1)[0, 0]
    film = torch.clamp(noise() - 0.25, min=0.0) * 0.03
    h = torch.maximum(film, plain - 0.9 + noise() - z)
    u, v = ((noise() - 0.5) * 1.6 * torch.clamp(h / 0.3, max=1.0) for _ in range(2))
    h, hu, hv = (a.to(dtype) for a in (h, h * u, h * v))
    sf = None if storage is None else (storage * noise()).to(dtype)
    return h, hu, hv, sf, (0.01 * noise()).to(dtype)


def _channel_state(net, slot, seed):
    """Wetted areas from half empty to just over the bank (below it where the slot above the
    bank is narrow), and downstream discharges."""
    tp = build_topology(net)
    sec = sections(tp, slot)
    r = np.random.default_rng([seed, 7])
    smooth = lambda: np.interp(np.arange(tp.n_cells), np.linspace(0, tp.n_cells, 12), r.uniform(0.0, 1.0, 12))
    y = sec["yb"] * (0.45 + (0.65 if slot > 0.1 else 0.4) * smooth())
    yt = np.minimum(y, sec["yb"])
    A = yt * (sec["b"] + sec["m"] * yt) + sec["ts"] * np.maximum(y - sec["yb"], 0.0)
    return A, A * (0.2 + smooth()) * (tp.kind != 1)


def _cfg(case, storm=None):
    cfg = SolverConfig(spatial_order=case.get("order", 2), flux=case.get("flux", "hllc"))
    if storm is not None:
        cfg.slot_width_frac = storm.slot_width_frac
    return cfg


def _dtype(case):
    return getattr(torch, case["dtype"])


def _grid_inputs(case, seed):
    """Fields and state of a grid case, in its precision."""
    ter = _terrain(case["nx"], case["ny"], case["dx"])
    dt, B = _dtype(case), case["members"]
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    full = lambda lo, hi: (lo + (hi - lo) * torch.rand(B, case["ny"], case["nx"], generator=g, device="cuda",
                                                       dtype=torch.float64)).to(dt)
    f = {"z": torch.as_tensor(ter.z, device="cuda").to(dt), "n": full(0.02, 0.06)}
    f["storage"] = full(0.0, 0.01) if case["sources"] else None
    f["horton"] = [full(30 * W.MMH, 90 * W.MMH), full(4 * W.MMH, 12 * W.MMH), full(2 / 3600, 6 / 3600)] \
        if case["sources"] else None
    f["weight"] = full(0.5, 1.5)[0] if case["weights"] else None
    h, hu, hv, sf, ic = _flooded(ter, B, seed, dt, f["storage"])
    return f, {"h": h, "hu": hu, "hv": hv, "sf": sf if sf is not None else torch.zeros_like(h), "ic": ic}


def _edges(case):
    val = {"S": SEA_LEVEL, "D": EDGE_INFLOW}
    return {e: EdgeBC(KIND_OF[k], val.get(k)) for e, k in zip(EDGES, case["edges"])}


def _coupled_inputs(case, seed):
    """Storms, 2-D state (members stacked) and channel states of a coupled case."""
    storms = _storms(case["nx"], case["ny"], case["dx"], case["members"], seed)
    S = torch.as_tensor(np.stack([s.storage for s in storms]), device="cuda")
    st = _flooded(storms[0].terrain, len(storms), seed, _dtype(case), S)
    chan = [_channel_state(s.network, s.slot_width_frac, seed + 31 * b) for b, s in enumerate(storms)]
    return storms, dict(zip(("h", "hu", "hv", "sf", "ic"), st)), np.stack([c[0] for c in chan]), np.stack([c[1] for c in chan])


def _groups(case):
    out = []
    for part in case["grids"].split(","):
        size, rest = part.split("@")
        dx, k = rest.split("*")
        out.append((int(size.split("x")[0]), int(size.split("x")[1]), float(dx), int(k)))
    return out


def _resident_inputs(case, seed):
    """One (storms, 2-D state, A, Q) per grid size of a resident case."""
    return [_coupled_inputs(dict(nx=nx, ny=ny, dx=dx, members=k, dtype=case["dtype"]), seed + 101 * j)
            for j, (nx, ny, dx, k) in enumerate(_groups(case))]


# --------------------------------------------------------------------------- the passes
def prepare(case, seed):
    kind, dt = case["kind"], _dtype(case)
    if kind == "grid":
        f, st = _grid_inputs(case, seed)
        B = case["members"]
        horton = Horton(*f["horton"], 0.0) if f["horton"] is not None else None
        one = lambda a: a if a is None or B > 1 else a[0]
        if horton is not None and B == 1:
            horton = Horton(*(a[0] for a in f["horton"]), 0.0)
        two = SWE2D(f["z"], one(f["n"]), case["dx"], _cfg(case), _edges(case), dtype=dt, storage=one(f["storage"]),
                    horton=horton, rain_weight=f["weight"], batch=B if B > 1 else None)
        two.set_state(*(one(st[k]) for k in ("h", "hu", "hv")))
        two.s_filled, two.infil_cum = one(st["sf"]), one(st["ic"])
        return {"case": case, "two": two, "t": 600.0}
    if kind == "resident":
        members, zcache = [], {}
        for storms, st, A, Q in _resident_inputs(case, seed):
            for b, s in enumerate(storms):
                m = Member(s, dt, torch.device("cuda", torch.cuda.current_device()), True, case["peaks"], zcache)
                for name, key in (("h", "h"), ("hu", "hu"), ("hv", "hv"), ("s_filled", "sf"), ("infil_cum", "ic")):
                    getattr(m, name).copy_(st[key][b])
                m.A.copy_(torch.as_tensor(A[b]))
                m.Q.copy_(torch.as_tensor(Q[b]))
                if case["peaks"]:
                    m.peak_h.copy_(m.h)
                members.append(m)
        cfg = SolverConfig(slot_width_frac=members[0].storm.slot_width_frac)
        eng = FloodEngine(members, cfg, "fp64" if dt == torch.float64 else "fp32", tile=(58, case["tile_y"]))
        eng.prepare(case["steps"])
        return {"case": case, "eng": eng}
    storms, st, A, Q = _coupled_inputs(case, seed)
    B = len(storms)
    pick = lambda a: a if B > 1 else a[0]
    if kind == "channel":
        f = [s.forcing for s in storms]
        bf = W.BatchForcing(f)
        one = SWE1D([s.network for s in storms] if B > 1 else storms[0].network, _cfg(case, storms[0]),
                    inflow=bf.inflow if B > 1 else f[0].inflow, stage=bf.tide if B > 1 else f[0].tide)
        one.A, one.Q = pick(A), pick(Q)
        return {"case": case, "one": one, "t": 0.0}
    if kind == "weir":
        cfg, ter = _cfg(case, storms[0]), storms[0].terrain
        two = SWE2D(ter.z, 0.03, ter.dx, cfg, {e: EdgeBC() for e in EDGES}, dtype=dt, batch=B if B > 1 else None)
        one = SWE1D([s.network for s in storms] if B > 1 else storms[0].network, cfg)
        two.set_state(pick(st["h"]), pick(st["hu"]), pick(st["hv"]))
        one.A, one.Q = pick(A), pick(Q)
        links = links_from_cells(one, two, *_bank_links(case["nx"], case["ny"], case["dx"]))
        return {"case": case, "one": one, "two": two, "links": links, "cfg": cfg}
    eng = build_engine_batch(storms, dtype=dt) if B > 1 else build_engine(storms[0], dtype=dt)
    eng.two.set_state(pick(st["h"]), pick(st["hu"]), pick(st["hv"]))
    eng.two.s_filled, eng.two.infil_cum = pick(st["sf"]), pick(st["ic"])
    eng.one.A, eng.one.Q = pick(A), pick(Q)
    return {"case": case, "eng": eng, "t": 0.0, "t_end": storms[0].t_end}


def _out2(two):
    return {"h": two.h, "hu": two.hu, "hv": two.hv, "s_filled": two.s_filled, "infil_cum": two.infil_cum}


def run(state):
    case = state["case"]
    kind, dt = case["kind"], _dtype(case)
    if kind == "grid":
        two = state["two"]
        step = two.max_dt()
        vols = two.step(step, state["t"], RAIN)
        state["t"] += step
        return dict(_out2(two), volumes=vols.table.to(dt))      # totals of the case's precision
    if kind == "channel":
        one = state["one"]
        n_sub = max(1, math.ceil(case["span"] / one.max_dt() - 1e-9))
        vols = one.substeps(case["span"], state["t"], n_sub)
        state["t"] += case["span"]
        return {"A": one.A, "Q": one.Q, "volumes": vols.table}
    if kind == "weir":
        one, two = state["one"], state["two"]
        V = exchange(one, two, state["links"], WEIR_DT, state["cfg"])
        return {"h": two.h, "hu": two.hu, "hv": two.hv, "A": one.A.to(dt), "V": V.to(dt)}
    eng = state["eng"]
    if kind == "coupled":
        state["t"] = eng.step(state["t"], state["t_end"])
        return dict(_out2(eng.two), A=eng.one.A.to(dt), Q=eng.one.Q.to(dt))
    eng.advance(case["steps"])
    flat = lambda name: torch.cat([getattr(m, name).reshape(-1) for m in eng.members])
    names = ["h", "hu", "hv", "s_filled", "infil_cum"] + (["peak_h", "peak_speed"] if case["peaks"] else [])
    return dict({k: flat(k) for k in names}, A=flat("A").to(dt), Q=flat("Q").to(dt))


# ------------------------------------------------------------------------ work of a pass
def _grid_work(cells, size, order, sources, weights=False, peaks=False, n=1):
    """Per step: state, bed and roughness read, state written; retention and infiltration
    fields and their state; the operations of one or two stages (two reconstructions, two
    faces and the limiter per cell) and of the sources."""
    vals = 5 + 3 + (8 if sources else 0) + (1 if weights else 0) + (4 if peaks else 0)
    return {"bytes": n * cells * vals * size, "flops": n * cells * ((2 * 230 if order == 2 else 130) + 60)}


def _channel_work(cells, n_sub, n=1):
    return {"bytes": n * cells * 8 * (4 + 9), "flops": n * cells * n_sub * 150}


def _weir_work(links, size):
    return {"bytes": links * (3 * size + 3 * 4 + 6 * size + 8), "flops": links * 40}


def _add(*parts):
    return {k: float(sum(p[k] for p in parts)) for k in ("bytes", "flops")}


def work(case):
    kind, size = case["kind"], 8 if case["dtype"] == "float64" else 4
    if kind == "resident":
        parts = []
        for nx, ny, dx, k in _groups(case):
            links = len(_bank_links(nx, ny, dx)[0])
            cells1 = build_topology(_network(_terrain(nx, ny, dx), 1.0)).n_cells
            n = k * case["steps"]
            parts += [_grid_work(nx * ny, size, 2, True, peaks=case["peaks"], n=n), _channel_work(cells1, 1, n),
                      _weir_work(links * n, size)]
        return _add(*parts)
    cells = case["nx"] * case["ny"] * case["members"]
    if kind == "grid":
        return _add(_grid_work(cells, size, case["order"], case["sources"], case["weights"]))
    B = case["members"]
    cells1 = B * build_topology(_network(_terrain(case["nx"], case["ny"], case["dx"]), 1.0)).n_cells
    if kind == "channel":
        return _add(_channel_work(cells1, max(1, round(case["span"] / 4.0))))
    links = _weir_work(B * len(_bank_links(case["nx"], case["ny"], case["dx"])[0]), size)
    if kind == "weir":
        return _add(links)
    return _add(_grid_work(cells, size, 2, True), _channel_work(cells1, 1), links)


# --------------------------------------------- the method in float64, as plain torch ops
class _Grid64:
    """Members of one grid size on the plain second- or first-order 2-D scheme: MUSCL with
    minmod, hydrostatic reconstruction, HLL/HLLC, outflow limiter, SSP-RK2, sources."""

    def __init__(self, z, n, dx, cfg, edges, storage=None, horton=None, weight=None):
        self.z, self.n, self.dx, self.cfg, self.edges = z, n, dx, cfg, edges
        self.storage, self.horton, self.weight = storage, horton, weight

    def velocity(self, h, hu, hv):
        h4 = h ** 4
        s = math.sqrt(2.0) * h / torch.sqrt(h4 + torch.clamp(h4, min=self.cfg.kp_eps))
        wet = h >= self.cfg.h_dry
        return torch.where(wet, hu * s, 0.0), torch.where(wet, hv * s, 0.0)

    def rate(self, h, hu, hv):
        u, v = self.velocity(h, hu, hv)
        c = torch.sqrt(self.cfg.g * h)
        r = (u.abs() + c) / self.dx + (v.abs() + c) / self.dx
        return torch.where(h > self.cfg.h_dry, r, 0.0).amax(dim=(-2, -1))

    def ghosts(self, kind, val, h, un, ut, z, far):
        """Two ghost layers beyond an edge from the layers inside it (nearest first): depth and
        outward-normal and tangential velocity; ``val`` is the edge's value per member."""
        g, dry = self.cfg.g, self.cfg.h_dry
        if kind in "TC":
            pick = [0, far]
            return [(h[k], -un[k] if kind == "C" else un[k], ut[k], z[k]) for k in pick]
        h, un, ut, z = h[0], un[0], ut[0], z[0]
        if kind == "S":
            hg = torch.clamp(val - z, min=0.0)
            ci, cg = torch.sqrt(g * h), torch.sqrt(g * hg)
            wet = h >= dry
            ug = torch.where(wet, un + 2.0 * (ci - cg), torch.zeros_like(un))
            fast = wet & (un > ci)
            ug, hg = torch.where(fast, un, ug), torch.where(fast, h, hg)
            ug = torch.where(hg >= dry, ug, torch.zeros_like(ug))
            ghost = (hg, ug, torch.where(ug > 0, ut, torch.zeros_like(ut)), z)
        else:
            hc = torch.clamp((val * val / g) ** (1.0 / 3.0), min=dry)
            hg = torch.where(h >= dry, h, hc.expand_as(h))
            ghost = (hg, -val / hg, torch.zeros_like(h), z)
        return [ghost, ghost]

    def sweep(self, h, un, ut, lo, hi, vlo, vhi):
        """Fluxes along the last axis: mass, momentum with the left and right pressure terms,
        tangential, at the n + 1 faces; and the bed term of the n cells."""
        cfg, z = self.cfg, self._z
        n = h.shape[-1]
        layer = lambda a, k: a[..., k]
        far = 1 if n > 1 else 0
        low = self.ghosts(lo, vlo, [layer(h, 0), layer(h, far)], [-layer(un, 0), -layer(un, far)],
                          [layer(ut, 0), layer(ut, far)], [layer(z, 0), layer(z, far)], far)
        high = self.ghosts(hi, vhi, [layer(h, n - 1), layer(h, n - 1 - far)], [layer(un, n - 1), layer(un, n - 1 - far)],
                           [layer(ut, n - 1), layer(ut, n - 1 - far)], [layer(z, n - 1), layer(z, n - 1 - far)], far)
        pad = lambda a, k, sl: torch.cat([sl * low[1][k][..., None], sl * low[0][k][..., None], a, high[0][k][..., None],
                                          high[1][k][..., None]], dim=-1)
        h, un, ut, z = pad(h, 0, 1.0), pad(un, 1, -1.0), pad(ut, 2, 1.0), pad(z, 3, 1.0)
        if cfg.spatial_order == 2:
            def minmod(a):
                l, r = a[..., 1:-1] - a[..., :-2], a[..., 2:] - a[..., 1:-1]
                m = torch.minimum(l.abs(), r.abs())
                return torch.where(l * r > 0, torch.where(l > 0, m, -m), torch.zeros_like(m)) * ok
            ok = (torch.minimum(torch.minimum(h[..., :-2], h[..., 1:-1]), h[..., 2:]) >= cfg.h_dry).double()
            half = [0.5 * minmod(a) for a in (h, un, ut, h + z)]
            mid = [a[..., 1:-1] for a in (h, un, ut, h + z)]
            minus, plus = [a - s for a, s in zip(mid, half)], [a + s for a, s in zip(mid, half)]
            zm, zp = minus[3] - minus[0], plus[3] - plus[0]
            bed = (-0.5 * cfg.g * (minus[0] + plus[0]) * (zp - zm))[..., 1:-1]
        else:
            minus = plus = [a[..., 1:-1] for a in (h, un, ut)]
            zm = zp = z[..., 1:-1]
            bed = None
        hL, uL, vL, zL = plus[0][..., :-1], plus[1][..., :-1], plus[2][..., :-1], zp[..., :-1]
        hR, uR, vR, zR = minus[0][..., 1:], minus[1][..., 1:], minus[2][..., 1:], zm[..., 1:]
        zf = torch.maximum(zL, zR)
        sL, sR = torch.clamp(hL + zL - zf, min=0.0), torch.clamp(hR + zR - zf, min=0.0)
        F1, F2, F3 = self.riemann(sL, uL, vL, sR, uR, vR)
        hg = 0.5 * cfg.g
        return F1, F2 + hg * (hL * hL - sL * sL), F2 + hg * (hR * hR - sR * sR), F3, bed

    def riemann(self, hL, uL, vL, hR, uR, vR):
        g, tiny = self.cfg.g, 1e-14
        cL, cR = torch.sqrt(g * hL), torch.sqrt(g * hR)
        dL, dR = hL <= tiny, hR <= tiny
        us, cs = 0.5 * (uL + uR) + cL - cR, 0.5 * (cL + cR) + 0.25 * (uL - uR)
        SL, SR = torch.minimum(uL - cL, us - cs), torch.maximum(uR + cR, us + cs)
        SL, SR = torch.where(dL, uR - 2 * cR, SL), torch.where(dL, uR + cR, SR)
        SL, SR = torch.where(dR, uL - cL, SL), torch.where(dR, uL + 2 * cL, SR)
        qL, qR = hL * uL, hR * uR
        pL, pR = qL * uL + 0.5 * g * hL * hL, qR * uR + 0.5 * g * hR * hR
        den = SR - SL
        den = torch.where(den.abs() < tiny, torch.ones_like(den), den)
        left, right = SL >= 0, SR <= 0
        hll = lambda a, b, qa, qb: torch.where(left, a, torch.where(right, b, (SR * a - SL * b + SL * SR * (qb - qa)) / den))
        F1, F2 = hll(qL, qR, hL, hR), hll(pL, pR, qL, qR)
        if self.cfg.flux == "hllc":
            dd = hR * (uR - SR) - hL * (uL - SL)
            SM = torch.where(dd.abs() < tiny, 0.5 * (uL + uR), (SL * hR * (uR - SR) - SR * hL * (uL - SL)) /
                             torch.where(dd.abs() < tiny, torch.ones_like(dd), dd))
            F3 = F1 * torch.where(SM >= 0, vL, vR)
        else:
            F3 = hll(qL * vL, qR * vR, hL * vL, hR * vR)
        both = dL & dR
        return tuple(torch.where(both, torch.zeros_like(f), f) for f in (F1, F2, F3))

    def tendency(self, h, hu, hv, dt, vals):
        """d(h, hu, hv)/dt with the limited fluxes, and the boundary in- and outflow."""
        dx = self.dx
        u, v = self.velocity(h, hu, hv)
        W_, E_, S_, N_ = self.edges
        edge = lambda k: vals[:, k, None]
        self._z = self.z.expand_as(h)
        X1, X2l, X2r, X3, bx = self.sweep(h, u, v, W_, E_, edge(0), edge(1))
        T = lambda a: a.transpose(-1, -2)
        self._z = T(self.z.expand_as(h))
        Y = self.sweep(T(h), T(v), T(u), S_, N_, edge(2), edge(3))
        Y1, Y2l, Y2r, Y3 = (T(a) for a in Y[:4])
        by = None if Y[4] is None else T(Y[4])
        relu = lambda a: torch.clamp(a, min=0.0)
        out = (relu(X1[..., 1:]) + relu(-X1[..., :-1])) / dx + (relu(Y1[..., 1:, :]) + relu(-Y1[..., :-1, :])) / dx
        need = out * dt
        th = torch.where(need > h, h / torch.where(need > 0, need, torch.ones_like(need)), torch.ones_like(need))
        ox, oy = torch.ones_like(th[..., :1]), torch.ones_like(th[..., :1, :])
        sx = torch.where(X1 > 0, torch.cat([ox, th], -1), torch.cat([th, ox], -1))
        sy = torch.where(Y1 > 0, torch.cat([oy, th], -2), torch.cat([th, oy], -2))
        X1, X3, Y1, Y3 = X1 * sx, X3 * sx, Y1 * sy, Y3 * sy
        d = lambda a: -(a[..., 1:] - a[..., :-1]) / dx
        e = lambda a: -(a[..., 1:, :] - a[..., :-1, :]) / dx
        dh = d(X1) + e(Y1)
        dhu = -(X2l[..., 1:] - X2r[..., :-1]) / dx + e(Y3)
        dhv = d(X3) - (Y2l[..., 1:, :] - Y2r[..., :-1, :]) / dx
        if bx is not None:
            dhu, dhv = dhu + bx / dx, dhv + by / dx
        qin = (relu(X1[..., 0]) + relu(-X1[..., -1])).sum(-1) + (relu(Y1[..., 0, :]) + relu(-Y1[..., -1, :])).sum(-1)
        qout = (relu(-X1[..., 0]) + relu(X1[..., -1])).sum(-1) + (relu(-Y1[..., 0, :]) + relu(Y1[..., -1, :])).sum(-1)
        return dh, dhu, dhv, qin * dx, qout * dx

    def step(self, st, dt, t, rain, vals0, vals1):
        """One step of every member with its own dt, clock and rain (B,); returns the volume
        table (boundary in, out, rain, infiltration, clip)."""
        cfg, area = self.cfg, self.dx * self.dx
        h, hu, hv = st["h"], st["hu"], st["hv"]
        D = dt[:, None, None]
        dh, dhu, dhv, qin, qout = self.tendency(h, hu, hv, D, vals0)
        h1, hu1, hv1 = h + D * dh, hu + D * dhu, hv + D * dhv
        neg = torch.clamp(-h1, min=0.0)
        clip = neg.sum((-2, -1)) * area
        h1 = h1 + neg
        if cfg.spatial_order == 2:
            dh, dhu, dhv, qin2, qout2 = self.tendency(h1, hu1, hv1, D, vals1)
            h1, hu1, hv1 = 0.5 * (h + h1 + D * dh), 0.5 * (hu + hu1 + D * dhu), 0.5 * (hv + hv1 + D * dhv)
            neg = torch.clamp(-h1, min=0.0)
            clip = clip + neg.sum((-2, -1)) * area
            h1, qin, qout = h1 + neg, 0.5 * (qin + qin2), 0.5 * (qout + qout2)
        h, hu, hv = h1, hu1, hv1
        add = (rain * dt)[:, None, None] * (self.weight if self.weight is not None else torch.ones_like(h[0]))
        h = h + add
        infil = torch.zeros_like(h)

        def lose(h, hu, hv, take):
            keep = torch.where(h > 0, (h - take) / torch.where(h > 0, h, torch.ones_like(h)), torch.zeros_like(h))
            return h - take, hu * keep, hv * keep
        if self.horton is not None:
            f0, fc, k = self.horton
            pot = (fc + (f0 - fc) * torch.exp(-k * torch.clamp(t, min=0.0)[:, None, None])) * D
            infil = torch.minimum(pot, h)
            h, hu, hv = lose(h, hu, hv, infil)
            if self.storage is not None:
                more = torch.minimum(pot - infil, st["sf"])
                st["sf"], infil = st["sf"] - more, infil + more
            st["ic"] = st["ic"] + infil
        if self.storage is not None:
            fill = torch.minimum(torch.clamp(self.storage - st["sf"], min=0.0), h)
            h, hu, hv = lose(h, hu, hv, fill)
            st["sf"] = st["sf"] + fill
        u, v = self.velocity(h, hu, hv)
        den = 1.0 + D * cfg.g * self.n * self.n * torch.sqrt(u * u + v * v) / torch.clamp(h, min=cfg.h_dry) ** (4.0 / 3.0)
        wet = h >= cfg.h_dry
        st["h"], st["hu"], st["hv"] = h, torch.where(wet, h * u / den, 0.0), torch.where(wet, h * v / den, 0.0)
        tot = lambda a: a.expand_as(h).sum((-2, -1)) * area
        return torch.stack([qin * dt, qout * dt, tot(add), tot(infil), clip], dim=1)


class _Channel64:
    """The members' channel networks: trapezoidal sections with a wall above the bank, HLL with
    hydrostatic reconstruction, outflow limiter, semi-implicit friction."""

    def __init__(self, nets, slot, cfg):
        tps = [build_topology(n) for n in nets]
        tp = tps[0]
        self.cfg = cfg
        D = lambda a: torch.as_tensor(np.array(a), device="cuda", dtype=torch.float64)
        I = lambda a: torch.as_tensor(np.array(a), device="cuda", dtype=torch.int64)
        secs = [sections(p, slot) for p in tps]
        self.s = {k: D(np.stack([s[k] for s in secs])) for k in secs[0]}
        self.z, self.bank = D(np.stack([p.z for p in tps])), D(tp.zbank)
        self.n, self.dx, self.sign = D(tp.n), D(tp.dx), D(tp.ghost_sign)
        self.kind, self.fl, self.fr = I(tp.kind), I(tp.face_l), I(tp.face_r)
        self.src = I(np.maximum(tp.ghost_src, 0))
        self.cell = [self.s[k] for k in ("b", "m", "yb", "ts")]
        self.face = [self.s[k] for k in ("fb", "fm", "fyb", "fts")]

    @staticmethod
    def area(s, y):
        b, m, yb, ts = s
        yt = torch.minimum(y, yb)
        return yt * (b + m * yt) + ts * torch.clamp(y - yb, min=0.0)

    @staticmethod
    def top(s, y):
        b, m, yb, ts = s
        return torch.where(y <= yb, b + 2 * m * y, ts)

    @staticmethod
    def moment(s, y):
        b, m, yb, ts = s
        yt, above = torch.minimum(y, yb), torch.clamp(y - yb, min=0.0)
        return b * yt * yt / 2 + m * yt ** 3 / 3 + yt * (b + m * yt) * above + ts * above * above / 2

    @staticmethod
    def depth(s, A):
        b, m, yb, ts = s
        A = torch.clamp(A, min=0.0)
        ab = yb * (b + m * yb)
        return torch.where(A <= ab, 2 * A / (b + torch.sqrt(b * b + 4 * m * A)), yb + (A - ab) / ts)

    def velocity(self, A, Q):
        return torch.where(self.depth(self.cell, A) >= self.cfg.h_dry, Q / torch.clamp(A, min=1e-12), 0.0)

    def rate(self, A, Q):
        """Largest wave rate over the wet interior cells, per member (0: none wet)."""
        y = self.depth(self.cell, A)
        on = (self.kind <= 1) & (y > self.cfg.h_dry)
        r = (self.velocity(A, Q).abs() + torch.sqrt(self.cfg.g * A / self.top(self.cell, y))) / self.dx
        return torch.where(on, r, 0.0).amax(-1)

    def substep(self, A, Q, dt, q_in, eta):
        cfg, kind, s = self.cfg, self.kind, self.cell
        g, dry = cfg.g, cfg.h_dry
        dt, q_in, eta = dt[:, None], q_in[:, None], eta[:, None]
        As, Qs = A[:, self.src], Q[:, self.src]
        ys = self.depth(s, As)
        wet = ys >= dry
        un = self.sign * torch.where(wet, Qs / torch.clamp(As, min=1e-12), 0.0)
        yst = torch.clamp(eta - self.z, min=0.0)
        Ast = self.area(s, yst)
        ci, cg = torch.sqrt(g * As / self.top(s, ys)), torch.sqrt(g * Ast / self.top(s, yst))
        ust = torch.where(wet, un + 2 * (ci - cg), 0.0)
        fast = wet & (un > ci)
        ust, Ast = torch.where(fast, un, ust), torch.where(fast, As, Ast)
        ust = torch.where(self.depth(s, Ast) >= dry, ust, 0.0)
        yc = torch.clamp((q_in * q_in / (g * s[0] * s[0])) ** (1.0 / 3.0), min=dry)
        A = torch.where(kind == 3, Ast, torch.where(kind == 2, torch.where(wet, As, self.area(s, yc)),
                                                    torch.where(kind == 4, As, A)))
        Q = torch.where(kind == 3, self.sign * Ast * ust, torch.where(kind == 2, -self.sign * q_in,
                                                                      torch.where(kind == 4, -Qs, Q)))
        y, u = self.depth(s, A), self.velocity(A, Q)
        f, l, r = self.face, self.fl, self.fr
        zf = torch.maximum(self.z[:, l], self.z[:, r])
        yL, yR = (torch.clamp(self.z[:, k] + y[:, k] - zf, min=0.0) for k in (l, r))
        AL, AR, uL, uR = self.area(f, yL), self.area(f, yR), u[:, l], u[:, r]
        pL, pR = g * self.moment(f, yL), g * self.moment(f, yR)
        cL, cR = torch.sqrt(g * AL / self.top(f, yL)), torch.sqrt(g * AR / self.top(f, yR))
        QL, QR = AL * uL, AR * uR
        dL, dR = AL <= 1e-14, AR <= 1e-14
        SL, SR = torch.minimum(uL - cL, uR - cR), torch.maximum(uL + cL, uR + cR)
        SL, SR = torch.where(dL, uR - 2 * cR, SL), torch.where(dL, uR + cR, SR)
        SL, SR = torch.where(dR, uL - cL, SL), torch.where(dR, uL + 2 * cL, SR)
        den = SR - SL
        den = torch.where(den.abs() < 1e-14, torch.ones_like(den), den)
        hll = lambda a, b, qa, qb: torch.where(dL & dR, torch.zeros_like(a), torch.where(SL >= 0, a, torch.where(
            SR <= 0, b, (SR * a - SL * b + SL * SR * (qb - qa)) / den)))
        F1, F2 = hll(QL, QR, AL, AR), hll(QL * uL + pL, QR * uR + pR, QL, QR)
        gather = lambda idx, val: torch.zeros_like(A).index_add_(1, idx, val)
        relu = lambda a: torch.clamp(a, min=0.0)
        need = (gather(l, relu(F1)) + gather(r, relu(-F1))) * dt
        vol = A * self.dx
        th = torch.where(need > vol, vol / torch.where(need > 0, need, torch.ones_like(need)), torch.ones_like(need))
        ghost = kind >= 2
        th = torch.where(ghost, torch.ones_like(th), th)
        F1 = F1 * torch.where(F1 > 0, th[:, l], th[:, r])
        gl, gr = ghost[l].double(), ghost[r].double()
        vin = (relu(F1) * gl + relu(-F1) * gr).sum(-1) * dt[:, 0]
        vout = (relu(-F1) * gl + relu(F1) * gr).sum(-1) * dt[:, 0]
        A1 = A + dt * (gather(r, F1) - gather(l, F1)) / self.dx
        Q1 = Q + dt * (gather(r, F2 - pR) - gather(l, F2 - pL)) / self.dx
        neg = relu(-A1)
        clip = (neg * self.dx * (~ghost)).sum(-1)
        A1 = A1 + neg
        y1, Ac = self.depth(s, A1), torch.clamp(A1, min=1e-12)
        R = Ac / (s[0] + 2 * torch.minimum(y1, s[2]) * torch.sqrt(1 + s[1] * s[1]))
        Q1 = Q1 / (1 + dt * g * self.n * self.n * Q1.abs() / (Ac * torch.clamp(R, min=dry) ** (4.0 / 3.0)))
        Q1 = torch.where((y1 >= dry) & (kind != 1), Q1, 0.0)
        return torch.where(ghost, A, A1), torch.where(ghost, Q, Q1), torch.stack([vin, vout, clip], 1)

    def advance(self, A, Q, dt, n_sub, q_in, eta):
        """n_sub (B,) substeps of dt / n_sub; q_in and eta give the forcing at the times of
        substep k of every member."""
        tot = torch.zeros(len(A), 3, device="cuda", dtype=torch.float64)
        for k in range(int(n_sub.max())):
            a, q, v = self.substep(A, Q, dt / n_sub, q_in(k), eta(k))
            on = k < n_sub
            A, Q = torch.where(on[:, None], a, A), torch.where(on[:, None], q, Q)
            tot = tot + v * on[:, None]
        return A, Q, tot


def _weir64(grid, chan, st, A, dt, links, z2):
    """The weir exchange of every member (dt: (B,)); returns the new A and the volumes."""
    cfg = chan.cfg
    c1, c2, length = links
    area, B = grid.dx * grid.dx, len(A)
    c1, c2 = (torch.as_tensor(np.array(a), device="cuda", dtype=torch.int64) for a in (c1, c2))
    uq, inv = torch.unique(c2, return_inverse=True)
    flat = {k: st[k].reshape(B, -1) for k in ("h", "hu", "hv")}
    y = chan.depth(chan.cell, A)
    eta1 = (chan.z + y)[:, c1]
    hq = flat["h"][:, uq]
    eta2 = z2[c2] + hq[:, inv]
    up, dn = torch.maximum(eta1, eta2), torch.minimum(eta1, eta2)
    du, dd = torch.clamp(up - chan.bank[c1], min=0.0), torch.clamp(dn - chan.bank[c1], min=0.0)
    ratio = torch.where(du > 0, dd / torch.where(du > 0, du, torch.ones_like(du)), 0.0)
    q = cfg.weir_cw * length * du ** 1.5 * torch.clamp(1.0 - ratio ** 1.5, min=0.0) ** 0.385
    plan = (chan.top(chan.cell, y) * chan.dx)[:, c1]
    V = torch.minimum(q * dt[:, None], cfg.exchange_relax * (up - dn) / (1.0 / area + 1.0 / plan))
    into = eta2 > eta1
    take2 = torch.zeros_like(hq).index_add_(1, inv, torch.where(into, V, 0.0))
    take1 = torch.zeros_like(A).index_add_(1, c1, torch.where(into, 0.0, V))
    have2 = cfg.exchange_limit * hq * area
    b, m, yb, _ = chan.cell
    have1 = cfg.exchange_limit * torch.clamp(A - yb * (b + m * yb), min=0.0) * chan.dx
    cut = lambda tot, have: torch.where(tot > have, have / torch.where(tot > 0, tot, torch.ones_like(tot)), torch.ones_like(tot))
    V = torch.where(into, V * cut(take2, have2)[:, inv], -V * cut(take1, have1)[:, c1])
    new = hq - torch.zeros_like(hq).index_add_(1, inv, V) / area
    keep = torch.where(hq > 0, torch.clamp(new / torch.where(hq > 0, hq, torch.ones_like(hq)), max=1.0), 0.0)
    for k in flat:
        flat[k] = flat[k].clone()
    flat["h"][:, uq] = new
    for k in ("hu", "hv"):
        flat[k][:, uq] = flat[k][:, uq] * keep
    st.update({k: a.reshape(st[k].shape) for k, a in flat.items()})
    return A + torch.zeros_like(A).index_add_(1, c1, V) / chan.dx, V


def _dt64(cfg, rate):
    return torch.clamp(torch.where(rate > 0, cfg.cfl / torch.where(rate > 0, rate, torch.ones_like(rate)), cfg.dt_max),
                       cfg.dt_min, cfg.dt_max)


def _coupled64(case, storms, st, A, Q, steps, shared, peaks=False):
    """Coupled steps of storms on one terrain; shared: one dt and substep count for all."""
    s0, dt_ = storms[0], _dtype(case)
    cfg, ter, B = _cfg(case, s0), s0.terrain, len(storms)
    to = lambda a: torch.as_tensor(np.stack(a), device="cuda", dtype=torch.float64).to(dt_).double()
    full = lambda a: np.broadcast_to(np.asarray(a, float), (ter.ny, ter.nx))
    z = to([ter.z])[0]
    grid = _Grid64(z, to([full(s.manning) for s in storms]), ter.dx, cfg, "TTST", to([s.storage for s in storms]),
                   [to([s.horton[j] for s in storms]) for j in range(3)])
    chan = _Channel64([s.network for s in storms], s0.slot_width_frac, cfg)
    st = {k: a.double() for k, a in st.items()}
    A, Q = (torch.as_tensor(a, device="cuda") for a in (A, Q))
    links = _bank_links(ter.nx, ter.ny, ter.dx)
    t = np.zeros(B)
    at = lambda name, tt: torch.tensor([getattr(s.forcing, name)(x) for s, x in zip(storms, tt)], device="cuda",
                                       dtype=torch.float64)
    edge = lambda tt: torch.stack([torch.zeros(B, device="cuda", dtype=torch.float64)] * 2 + [at("tide", tt)] +
                                  [torch.zeros(B, device="cuda", dtype=torch.float64)], dim=1)
    pk, ps = st["h"].clone(), torch.zeros_like(st["h"])
    for _ in range(steps):
        r2, r1 = grid.rate(st["h"], st["hu"], st["hv"]), chan.rate(A, Q)
        if shared:
            r2, r1 = r2.max().expand(B), r1.max().expand(B)
        dt = _dt64(cfg, r2)
        dt1 = torch.where(r1 > 0, torch.clamp(cfg.cfl_1d / torch.where(r1 > 0, r1, torch.ones_like(r1)), max=cfg.dt_max),
                          cfg.dt_max)
        n_sub = torch.clamp(torch.ceil(dt / dt1 - 1e-9), min=1.0)
        A, _ = _weir64(grid, chan, st, A, dt, links, z.reshape(-1))
        d, n = dt.cpu().numpy(), n_sub.cpu().numpy()
        grid.step(st, dt, torch.as_tensor(t, device="cuda"), at("rain_rate", t), edge(t), edge(t + d))
        A, Q, _ = chan.advance(A, Q, dt, n_sub, lambda k: at("inflow", t + k * d / n), lambda k: at("tide", t + k * d / n))
        t = t + d
        u, v = grid.velocity(st["h"], st["hu"], st["hv"])
        pk, ps = torch.maximum(pk, st["h"]), torch.maximum(ps, torch.sqrt(u * u + v * v))
    out = {"h": st["h"], "hu": st["hu"], "hv": st["hv"], "s_filled": st["sf"], "infil_cum": st["ic"], "A": A, "Q": Q}
    return dict(out, peak_h=pk, peak_speed=ps) if peaks else out


def exact(case, seed):
    kind = case["kind"]
    if kind == "grid":
        f, st = _grid_inputs(case, seed)
        wide = lambda a: None if a is None else a.double()
        cfg, B = _cfg(case), case["members"]
        grid = _Grid64(wide(f["z"]), wide(f["n"]), case["dx"], cfg, case["edges"], wide(f["storage"]),
                       None if f["horton"] is None else [wide(a) for a in f["horton"]], wide(f["weight"]))
        st = {k: a.double() for k, a in st.items()}
        dt = _dt64(cfg, grid.rate(st["h"], st["hu"], st["hv"]).max()).expand(B)
        flat = lambda x: torch.full((B,), x, device="cuda", dtype=torch.float64)
        vals = torch.tensor([{"S": SEA_LEVEL, "D": EDGE_INFLOW}.get(k, 0.0) for k in case["edges"]], device="cuda",
                            dtype=torch.float64).expand(B, 4)
        vols = grid.step(st, dt, flat(600.0), flat(RAIN), vals, vals)
        one = lambda a: a if B > 1 else a[0]
        return {"h": one(st["h"]), "hu": one(st["hu"]), "hv": one(st["hv"]), "s_filled": one(st["sf"]),
                "infil_cum": one(st["ic"]), "volumes": vols}
    if kind == "resident":
        outs = [_coupled64(case, *part, case["steps"], False, case["peaks"]) for part in _resident_inputs(case, seed)]
        return {k: torch.cat([o[k].reshape(-1) for o in outs]) for k in outs[0]}
    storms, st, A, Q = _coupled_inputs(case, seed)
    B = len(storms)
    one = lambda a: a if B > 1 else a[0]
    if kind == "coupled":
        return {k: one(a) for k, a in _coupled64(case, storms, st, A, Q, 1, True).items()}
    cfg = _cfg(case, storms[0])
    chan = _Channel64([s.network for s in storms], storms[0].slot_width_frac, cfg)
    A, Q = (torch.as_tensor(a, device="cuda") for a in (A, Q))
    if kind == "weir":
        st = {k: a.double() for k, a in st.items()}
        z = torch.as_tensor(storms[0].terrain.z, device="cuda").to(_dtype(case)).double()
        grid = _Grid64(z, None, case["dx"], cfg, "TTTT")
        A, V = _weir64(grid, chan, st, A, torch.full((B,), WEIR_DT, device="cuda", dtype=torch.float64),
                       _bank_links(case["nx"], case["ny"], case["dx"]), z.reshape(-1))
        return {k: one(a) for k, a in dict(h=st["h"], hu=st["hu"], hv=st["hv"], A=A, V=V).items()}
    r = float(chan.rate(A, Q).max())
    n = max(1, math.ceil(case["span"] / (min(cfg.cfl_1d / r, cfg.dt_max) if r > 0 else cfg.dt_max) - 1e-9))
    full = lambda x: torch.full((B,), float(x), device="cuda", dtype=torch.float64)
    at = lambda name, k: torch.tensor([getattr(s.forcing, name)(k * case["span"] / n) for s in storms], device="cuda",
                                      dtype=torch.float64)
    A, Q, vols = chan.advance(A, Q, full(case["span"]), full(n), lambda k: at("inflow", k), lambda k: at("tide", k))
    return {"A": one(A), "Q": one(Q), "volumes": vols}
