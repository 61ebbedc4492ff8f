"""The work that users of this framework have it do, as measurable cases.

A case is a dict of plain values; `kind` says which public entry points it goes through:

  steps     FusedSolver.step on one catchment: the fused step (FP32 or FP64, either order)
  ensemble  FusedSolver on several catchments of mixed sizes, per-step launches or one
            persistent launch (run_persistent)
  coupled   the coupled server's exchange: 1st-order steps with an inflow edge, then depth and
            velocity at the agents' cells (ops.gather)
  gauges    one calibration pass: GaugeMisfit.simulate and .gradient (the adjoint)
  godunov   the reference's solver object over the drop-in ops, the server's loop
  host      HostStepper: the state in pinned host memory, copied in and out every step

Terrain is a seeded smooth random field, 50 m of relief over 4 km, with 10 m buildings on about
8 % of the cells, at the millimetre resolution elevation rasters have; water is a thin film with
ponds and moderate currents, the state a storm leaves after its first minutes.  `exact` evaluates
the same scheme on the dense raster in 64 bits with torch.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "chans-hipims-flamegpu_b200"))

from hipims_b200 import ops  # noqa: E402
from hipims_b200.adjoint import GaugeMisfit  # noqa: E402
from hipims_b200.fused import Catchment, FusedSolver, HostStepper  # noqa: E402
from hipims_b200.solver import Godunov  # noqa: E402

HS, G = 1.0e-6, 9.81          # the scheme's dry depth and gravity
MM_PER_H = 1.0e-3 / 3600.0    # m/s per mm/h
FOREVER = 1.0e9               # end of the rain and boundary tables (s)
DTYPES = {"f32": torch.float32, "f64": torch.float64}
OPEN, WALL, INFLOW = 50, 40, 70  # boundary codes: zero gradient, slip wall, given discharge


def listed():
    return [
        # the 256^2 dam break in a walled box every solver is first tried on: latency and launches
        dict(name="dam_break_256_f32", kind="steps", rows=256, cols=256, dtype="f32", order=2,
             terrain="flat", ring=WALL, sources=False, steps=16),
        # the urban storm on 2048^2 cells, the size production runs and the benchmark use
        dict(name="urban_2048_f32", kind="steps", rows=2048, cols=2048, dtype="f32", order=2,
             terrain="urban", ring=OPEN, sources=False, steps=16),
        # gauged rainfall and soils: station rain and Green-Ampt infiltration, ragged raster
        dict(name="stations_soils_f32", kind="steps", rows=1000, cols=1413, dtype="f32", order=2,
             terrain="urban", ring=OPEN, sources=True, steps=8),
        # double precision, as reference runs and calibrations use it
        dict(name="urban_1024_f64", kind="steps", rows=1024, cols=1024, dtype="f64", order=2,
             terrain="urban", ring=OPEN, sources=False, steps=8),
        # double precision, 1st order, a small odd catchment
        dict(name="village_f64_o1", kind="steps", rows=301, cols=517, dtype="f64", order=1,
             terrain="urban", ring=OPEN, sources=False, steps=8),
        # a storm ensemble: many catchments of mixed sizes, a launch per step
        dict(name="ensemble_f32", kind="ensemble", count=16, lo=128, hi=768, persistent=False,
             steps=16),
        # a smaller ensemble advanced by one persistent launch
        dict(name="ensemble_persistent_f32", kind="ensemble", count=6, lo=160, hi=512,
             persistent=True, steps=20),
        # a city coupled to the agent model: 1st order, inflow hydrograph, agents' water read back
        dict(name="city_coupled_f32", kind="coupled", rows=3000, cols=4100, agents=100_000,
             steps=8),
        # calibration of Manning's n and the rain against gauges: forward and adjoint
        dict(name="calibration_f64", kind="gauges", rows=512, cols=512, steps=40, every=10,
             checkpoint=20),
        # a program written for the reference's solver object, double precision, 2nd order
        dict(name="solver_object_f64", kind="godunov", rows=1024, cols=1024, dtype="f64", order=2,
             steps=4),
        # the same loop at the coupled server's settings: single precision, 1st order, small
        dict(name="solver_object_f32_o1", kind="godunov", rows=256, cols=300, dtype="f32", order=1,
             steps=8),
        # a host program that owns the state and hands it over every step
        dict(name="host_state_f32", kind="host", rows=1024, cols=1024, steps=4),
    ]


def draw(rng):
    """One more case of the same ranges."""

    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["steps"] * 5 + ["ensemble", "coupled", "gauges", "godunov", "godunov",
                                       "host"])
    if kind == "steps":
        dtype = rng.choice(["f32", "f32", "f64"])
        top = 2048 if dtype == "f32" else 1024
        return dict(kind=kind, rows=size(100, top), cols=size(100, top), dtype=dtype,
                    order=rng.choice([1, 2, 2]), terrain=rng.choice(["flat", "urban", "urban"]),
                    ring=rng.choice([OPEN, WALL]), sources=rng.random() < 0.25,
                    steps=2 * rng.randint(2, 8))
    if kind == "ensemble":
        lo = size(100, 250)
        return dict(kind=kind, count=rng.randint(2, 16), lo=lo, hi=lo + size(50, 500),
                    persistent=rng.random() < 0.5, steps=2 * rng.randint(4, 10))
    if kind == "coupled":
        return dict(kind=kind, rows=size(300, 2500), cols=size(300, 3000),
                    agents=size(1000, 100_000), steps=2 * rng.randint(2, 4))
    if kind == "gauges":
        return dict(kind=kind, rows=size(100, 512), cols=size(100, 512),
                    steps=10 * rng.randint(2, 4), every=10, checkpoint=rng.choice([10, 20, 100]))
    if kind == "godunov":
        return dict(kind=kind, rows=size(100, 1024), cols=size(100, 1024),
                    dtype=rng.choice(["f32", "f64"]), order=rng.choice([1, 2]),
                    steps=rng.randint(2, 6))
    return dict(kind=kind, rows=size(200, 1024), cols=size(200, 1024), steps=rng.randint(2, 4))


# --------------------------------------------------------------------------- inputs
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _field(rows, cols, gen, power):
    """Smooth random field scaled to [0, 1]."""
    dev = _device()
    k = torch.sqrt(torch.fft.fftfreq(rows, device=dev, dtype=torch.float64)[:, None] ** 2 +
                   torch.fft.rfftfreq(cols, device=dev, dtype=torch.float64)[None, :] ** 2)
    amp = k.clamp_min(1.0 / (4 * max(rows, cols))) ** (-power / 2.0)
    noise = torch.randn(rows, cols, generator=gen, dtype=torch.float64, device=dev)
    f = torch.fft.irfft2(torch.fft.rfft2(noise) * amp, s=(rows, cols))
    return (f - f.min()) / (f.max() - f.min())


def _quant(x, bits=10):
    return torch.round(x * 2.0 ** bits) / 2.0 ** bits


def _inputs(case, seed, which=0):
    """Rasters (with a no-data ring) and settings of one catchment, float64 arrays whose values
    are exact in float32."""
    rows, cols = case["rows"], case["cols"]
    gen = torch.Generator(device=_device())
    gen.manual_seed(seed * 1009 + which * 7 + 13)
    rng = np.random.default_rng(seed * 1009 + which * 7 + 17)
    kind, terrain = case["kind"], case.get("terrain", "urban")
    ring = case.get("ring", OPEN)
    if terrain == "flat":
        z = torch.zeros(rows, cols, dtype=torch.float64, device=_device())
        level = float(rng.uniform(0.9, 1.1))
        # a dam across the box at a slant
        r = torch.arange(rows, device=z.device, dtype=torch.float64)[:, None] / rows - 0.5
        c = torch.arange(cols, device=z.device, dtype=torch.float64)[None, :] / cols - 0.5
        wet = c + rng.uniform(0.5, 0.9) * r < rng.uniform(-0.05, 0.05)
        h = torch.where(wet, level, 0.05) + 0.02 * _field(rows, cols, gen, 4.0)
        speed = 0.0
    else:
        # 50 m over 2048 cells, the same slopes on smaller rasters
        ground = 50.0 * max(rows, cols) / 2048.0 * _field(rows, cols, gen, 4.0)
        z = ground.clone()
        side = 18
        for _ in range(max(1, int(0.08 * rows * cols / (side * side)))):
            a, b = rng.integers(5, 31, 2)
            r, c = rng.integers(0, max(rows - a, 1)), rng.integers(0, max(cols - b, 1))
            z[r:r + a, c:c + b] = ground[r:r + a, c:c + b] + 10.0
        z = _quant(z)
        pond = 4.0 * (_field(rows, cols, gen, 4.0) - 0.5).clamp_min(0.0)
        h = torch.where(z > ground + 5.0, 0.0, pond) + 0.002 + 0.03 * _field(rows, cols, gen, 4.0)
        speed = 0.4
    h = _quant(h, 20).float().double()
    u = speed * (2.0 * _field(rows, cols, gen, 4.0) - 1.0)
    v = speed * (2.0 * _field(rows, cols, gen, 4.0) - 1.0)
    qx, qy = (h * u).float().double(), (h * v).float().double()
    zone = (_field(rows, cols, gen, 4.0) > 0.45)

    def pad(x, dtype):
        out = np.zeros((rows + 2, cols + 2), dtype=dtype)
        out[1:-1, 1:-1] = x.cpu().numpy()
        return out

    mask = np.full((rows + 2, cols + 2), 1, dtype=np.int32)
    mask[1, :] = mask[-2, :] = mask[:, 1] = mask[:, -2] = ring
    rate = 50.0 * MM_PER_H
    d = dict(z=pad(z, np.float64), h=pad(h, np.float64), qx=pad(qx, np.float64),
             qy=pad(qy, np.float64), zone=pad(zone, np.uint8), manning=[0.035, 0.08], dx=2.0,
             cfl=0.5, dt0=0.05, rain=np.array([[0.0, rate], [FOREVER, rate]]))
    if kind == "coupled":
        mask[1:-1, 1] = INFLOW
        d["given_q"] = np.array([[0.0, 0.05, 0.0], [FOREVER, 0.05, 0.0]])
    if kind == "ensemble":  # each its own storm
        times = np.linspace(0.0, 7200.0, 121)
        peak = rng.uniform(300.0, 1800.0)
        rates = rng.uniform(20.0, 120.0) * MM_PER_H * (0.1 + np.clip(
            1.0 - np.abs(times - peak) / 900.0, 0.0, None))
        d["rain"] = np.stack([np.append(times, FOREVER), np.append(rates, rates[-1])], 1)
    if kind == "gauges":
        zones = _field(rows, cols, gen, 4.0) * 0.999
        d["zone"] = pad((zones * 8).to(torch.uint8), np.uint8)
        d["manning"] = [float(x) for x in rng.uniform(0.02, 0.10, 8)]
        pick = np.sort(rng.choice(rows * cols, size=min(32, rows * cols), replace=False))
        d["gauge_rows"], d["gauge_cols"] = pick // cols + 1, pick % cols + 1
        d["obs"] = rng.uniform(0.0, 0.5, (case["steps"] // case["every"], pick.size))
    if case.get("sources"):
        n = 6
        station = (_field(rows, cols, gen, 4.0) * 0.999 * n).to(torch.int64)
        d["station"] = pad(station, np.int64)
        rates = rng.uniform(10.0, 90.0, (2, n)) * MM_PER_H
        d["rain"] = np.concatenate([np.array([[0.0], [3.0e4]]), rates], 1)
        d["rain"] = np.concatenate([d["rain"], [[FOREVER] + list(rates[1])]], 0)
        d["infiltration"] = dict(ks=[1.0e-6, 3.0e-6], psi=[0.1, 0.2], dtheta=[0.2, 0.3])
    mask[0, :] = mask[-1, :] = -9999
    mask[:, 0] = mask[:, -1] = -9999
    d["mask"] = mask
    return d


def _catchment(d, **over):
    kw = dict(mask=d["mask"], z=d["z"], h=d["h"], qx=d["qx"], qy=d["qy"], zone=d["zone"],
              manning=d["manning"], dx=d["dx"], cfl=d["cfl"], dt0=d["dt0"], rain=d["rain"],
              given_q=d.get("given_q"), infiltration=d.get("infiltration"),
              rain_station=d.get("station"))
    kw.update(over)
    return Catchment(**kw)


def _members(case, seed):
    """The ensemble's catchments: sides spread over [lo, hi]."""
    rng = np.random.default_rng(case["count"] * 31 + case["lo"])  # sizes belong to the case
    sides = rng.integers(case["lo"], case["hi"] + 1, size=(case["count"], 2))
    return [_inputs(dict(case, rows=int(r), cols=int(c)), seed, k)
            for k, (r, c) in enumerate(sides)]


def _agents(case, seed):
    rows, cols = case["rows"], case["cols"]
    rng = np.random.default_rng(seed + 65537)
    pick = np.sort(rng.integers(0, rows * cols, size=case["agents"]))
    return pick // cols + 1, pick % cols + 1


def _views(fs, buf):
    """The latest state's rasters: step() leaves it in buffer `buf`."""
    out = []
    for ins in fs.inst:
        out.append({"h": ins.raster(ins.h[buf]), "qx": ins.raster(ins.qx[buf]),
                    "qy": ins.raster(ins.qy[buf]), "h_max": ins.raster(ins.h_max)})
        if ins.cum is not None:
            out[-1]["cum"] = ins.raster(ins.cum)
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("steps", "coupled"):
        f32 = case.get("dtype", "f32") == "f32"
        s["fs"] = FusedSolver(_catchment(_inputs(case, seed)),
                              dtype=torch.float32 if f32 else torch.float64,
                              order=case.get("order", 1))
        if kind == "coupled":
            s["agents"] = s["fs"].cell_offsets(0, *_agents(case, seed))
    elif kind == "ensemble":
        s["fs"] = FusedSolver([_catchment(d) for d in _members(case, seed)])
    elif kind == "host":
        s["fs"] = FusedSolver(_catchment(_inputs(case, seed)))
        s["host"] = HostStepper(s["fs"])
    elif kind == "gauges":
        d = _inputs(case, seed)
        s["problem"] = GaugeMisfit(_catchment(d), d["gauge_rows"], d["gauge_cols"], case["steps"],
                                   np.full(case["steps"], d["dt0"]), every=case["every"],
                                   checkpoint=case["checkpoint"], obs=d["obs"])
        s["manning"] = [1.2 * n for n in d["manning"]]
    else:
        d = _inputs(case, seed)
        dev = torch.device("cuda")
        g = Godunov(dev, d["dx"], d["cfl"], FOREVER, secondOrder=case["order"] == 2,
                    firstTimeStep=d["dt0"], tensorType=DTYPES[case["dtype"]])
        mask = torch.as_tensor(d["mask"], device=dev)
        g.init__fluidField_tensor(mask, d["h"], d["qx"], d["qy"], d["h"] + d["z"], d["z"], dev)
        g.set_landuse(mask, d["zone"], dev)
        g.set__frictionField_tensor(torch.tensor(d["manning"], dtype=torch.float64, device=dev),
                                    dev)
        g.set_distributed_rainfall_station_Mask(mask, np.zeros(d["mask"].shape, np.int16), dev)
        s["solver"], s["rain"], s["dev"] = g, d["rain"], dev
    if "fs" in s and kind != "host":  # an even number of steps ends in the buffer it began in
        s["cur"] = s["fs"].controls()[0].cur
    return s


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind in ("steps", "ensemble", "coupled"):
        fs = state["fs"]
        if case.get("persistent"):
            fs.run_persistent(case["steps"])
        else:
            fs.step(case["steps"])
        out = _views(fs, state["cur"])
        if kind == "coupled":
            ins, cur = fs.inst[0], state["cur"]
            out.append(ops.gather(state["agents"], ins.h[cur], ins.qx[cur], ins.qy[cur],
                                  velocities=True))
        return out
    if kind == "host":
        for _ in range(case["steps"]):
            state["host"].step()
        state["host"].finish()
        return list(state["host"].out_buffers)
    if kind == "gauges":
        p = state["problem"]
        samples = p.simulate(state["manning"], 1.1)
        loss = p.loss()
        grad, initial = p.gradient(with_state=True)
        return {"samples": samples, "loss": loss, "grad": grad, "initial": initial}
    g, dev = state["solver"], state["dev"]
    for _ in range(case["steps"]):
        g.addFlux()
        g.addStation_PrecipitationSource(state["rain"], dev)
        g.time_friction_euler_update_cuda(dev)
    return {"h": g._h_internal, "qx": g._qx_internal, "qy": g._qy_internal,
            "wl": g._wl_internal, "h_max": g._h_max}


# Operations of one cell's step counted in the scheme: two faces (reconstruction, hydrostatic
# step, Riemann solver) and one update.
FLOPS = {1: 230, 2: 300}


def work(case):
    kind, steps = case["kind"], case["steps"]
    if kind == "ensemble":
        rng = np.random.default_rng(case["count"] * 31 + case["lo"])
        sides = rng.integers(case["lo"], case["hi"] + 1, size=(case["count"], 2))
        cells, order, size = int((sides[:, 0] * sides[:, 1]).sum()), 2, 4
    else:
        cells = case["rows"] * case["cols"]
        order = case.get("order", 1 if kind == "coupled" else 2)
        size = 8 if kind == "gauges" or case.get("dtype") == "f64" else 4
    # h, qx, qy, z, h_max and the cell code read; h, qx, qy, h_max written
    step = cells * (9 * size + 1)
    if case.get("sources"):
        step += cells * (2 + 2 * size)  # station id; infiltrated depth read and written
    if kind == "gauges":
        # forward once, and one reverse step: state, bed, code and adjoint read, adjoint written
        rev = cells * (10 * size + 1)
        return {"bytes": steps * (step + rev), "flops": steps * cells * FLOPS[2] * 4}
    total = steps * step
    if kind == "coupled":
        total += case["agents"] * (8 + 6 * size)
    if kind == "host":
        total += steps * cells * 6 * size  # h, qx, qy over the bus, in and out
    return {"bytes": total, "flops": steps * cells * FLOPS[order]}


# --------------------------------------------------------------------------- 64 bits
def _minmod(a, b):
    return torch.where(a * b <= 0.0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))


def _hydro(order, La, Lb, L, Lz, R, Rz):
    """Hydrostatic reconstruction: depths and beds of both edges."""
    hi, lo = torch.maximum(La, Lb), torch.minimum(La, Lb)
    lw = torch.maximum(torch.minimum(L + Lz, hi), lo)
    rw = torch.maximum(torch.minimum(R + Rz, hi), lo)
    if order == 2:
        top = torch.maximum(lw, rw)
        lw, rw = torch.where(La > Lb, top, lw), torch.where(La > Lb, rw, top)
    else:
        flip = (La - Lb) * (lw - rw) < 0.0
        mid = (lw + rw) / 2.0
        lw, rw = torch.where(flip, mid, lw), torch.where(flip, mid, rw)
    bed = torch.maximum(lw - L, rw - R)
    hl, hr = (lw - bed).clamp_min(0.0), (rw - bed).clamp_min(0.0)
    return hl, lw - hl, hr, rw - hr


def _hllc(hl, hr, ul, ur, vl, vr):
    """Mass, normal and tangential momentum flux."""
    al, ar = (G * hl).sqrt(), (G * hr).sqrt()
    us = (ul + ur) / 2.0 + al - ar
    ast = ((al + ar) / 2.0 + (ul - ur) / 4.0).abs()
    sl = torch.where(hl <= HS, ur - 2.0 * ar, torch.minimum(ul - al, us - ast))
    sr = torch.where(hr <= HS, ul + 2.0 * al, torch.maximum(ur + ar, us + ast))
    pl, pr = hl * (ul - sl), hr * (ur - sr)
    sm = (sl * pr - sr * pl) / (pr - pl)
    nl, nr = ul * ul * hl + 0.5 * G * hl * hl, ur * ur * hr + 0.5 * G * hr * hr
    fm = (sr * ul * hl - sl * ur * hr + sl * sr * (hr - hl)) / (sr - sl)
    nm = (sr * nl - sl * nr + sl * sr * (ur * hr - ul * hl)) / (sr - sl)
    left = sl >= 0.0
    ml = ~left & (sm >= 0.0)
    mr = ~left & (sm < 0.0) & (sr >= 0.0)
    mid = ml | mr
    f = torch.where(left, ul * hl, torch.where(mid, fm, ur * hr))
    n = torch.where(left, nl, torch.where(mid, nm, nr))
    t = f * torch.where(left | ml, vl, vr)
    dry = (hl < HS) & (hr < HS)
    zero = torch.zeros_like(f)
    return [torch.where(dry, zero, x) for x in (f, n, t)]


def _faces(order, A, B, AA, BB, vAA, vBB):
    """Faces between minus-side cells A and plus-side cells B (h, z, normal and tangential q);
    AA, BB the cells beyond, vAA, vBB whether they are valid.  Fluxes and both bed-slope terms."""
    own = [torch.where(vAA, x, a) for x, a in zip(AA, A)]
    far = [torch.where(vBB, x, b) for x, b in zip(BB, B)]
    sA = [0.5 * _minmod(a - o, b - a) for a, o, b in zip(A, own, B)]
    sB = [0.5 * _minmod(b - a, f - b) for a, f, b in zip(A, far, B)]
    zero = torch.zeros_like(A[0])
    if order == 2:
        L = [a + s for a, s in zip(A, sA)]
        R = [b - s for b, s in zip(B, sB)]
        for e, c in ((L, A), (R, B)):
            e[2], e[3] = torch.where(c[0] < HS, zero, e[2]), torch.where(c[0] < HS, zero, e[3])
    else:
        L, R = list(A), list(B)
        L[1] = torch.where(B[0] > HS, A[1] + sA[1], A[1])
        R[1] = torch.where(A[0] > HS, B[1] - sB[1], B[1])
    return _edge_flux(order, A, B, L, R)


def _edge_flux(order, A, B, L, R):
    zero = torch.zeros_like(A[0])
    il = torch.where(L[0] < HS, zero, 1.0 / L[0])
    ir = torch.where(R[0] < HS, zero, 1.0 / R[0])
    hl, zl, hr, zr = _hydro(order, A[0] + A[1], B[0] + B[1], L[0], L[1], R[0], R[1])
    f = _hllc(hl, hr, L[2] * il, R[2] * ir, L[3] * il, R[3] * ir)
    sa = 0.5 * G * (A[0] + hl) * (zl - A[1])
    sb = 0.5 * G * (B[0] + hr) * (zr - B[1])
    dry = (A[0] < HS) & (B[0] < HS)
    return [torch.where(dry, zero, x) for x in (*f, sa, sb)]


class _Dense:
    """The scheme on a dense raster with a two-cell no-data margin, in 64 bits."""

    def __init__(self, d, order, manning=None, rain_mult=1.0):
        dev = _device()
        t = lambda a: torch.nn.functional.pad(  # noqa: E731
            torch.as_tensor(np.asarray(a, dtype=np.float64), device=dev), (1, 1, 1, 1))
        self.order, self.dev, self.d, self.mult = order, dev, d, rain_mult
        code = t(np.maximum(d["mask"], 0)).to(torch.int64)
        self.valid = code > 0
        self.h, self.z, self.qx, self.qy = t(d["h"]), t(d["z"]), t(d["qx"]), t(d["qy"])
        self.h_max = self.h.clone()
        zone = t(d["zone"]).to(torch.int64)
        n = d["manning"] if manning is None else manning
        self.n = torch.tensor(n, dtype=torch.float64, device=dev)[zone]
        self.dx, self.cfl, self.dt, self.t = d["dx"], d["cfl"], d["dt0"], 0.0
        first = torch.nonzero(self.valid.flatten())[0]
        self.counts = self.valid.clone()  # the first cell never activates its neighbours
        self.counts.view(-1)[first] = False
        self.cum = None
        if d.get("infiltration"):
            self.cum = torch.zeros_like(self.h)
            self.soil = {k: torch.tensor(v, dtype=torch.float64, device=dev)[zone]
                         for k, v in d["infiltration"].items()}
            self.station = t(d["station"]).to(torch.int64)
        # cells that miss a neighbour: (row offset, column offset) of E, N, W, S
        self.edges = []
        for dy, dx in ((0, 1), (-1, 0), (0, -1), (1, 0)):
            nb = torch.roll(self.valid, (-dy, -dx), (0, 1))
            rr, cc = torch.nonzero(self.valid & ~nb, as_tuple=True)
            kind = code[rr, cc]
            while bool((kind >= 10).any()):
                kind = torch.where(kind >= 10, kind // 10, kind)
            self.edges.append((dy, dx, rr, cc, kind))

    def _rain(self):
        R, t = self.d["rain"], self.t
        rates = [np.interp(t, R[:, 0], R[:, k]) if t < R[-1, 0] else 0.0
                 for k in range(1, R.shape[1])]
        rates = torch.tensor(rates, dtype=torch.float64, device=self.dev) * self.mult
        return rates[self.station] if self.cum is not None else rates[0]

    def _ghosts(self, dy, dx, rr, cc, kind):
        """Outward mass and x, y momentum flux and the bed-slope term (global axes)."""
        h, z = self.h[rr, cc], self.z[rr, cc]
        qx, qy = self.qx[rr, cc], self.qy[rr, cc]
        n0, n1 = float(dx), float(-dy)
        q = self.d.get("given_q")
        gqx = torch.where(kind == 4, (n1 * n1 - n0 * n0) * qx, qx)
        gqy = torch.where(kind == 4, (n0 * n0 - n1 * n1) * qy, qy)
        if q is not None:
            gqx = torch.where(kind == 7, torch.full_like(qx, q[0, 1]), gqx)
            gqy = torch.where(kind == 7, torch.full_like(qy, q[0, 2]), gqy)
        frame = lambda x, y: (x * n0 + y * n1, -x * n1 + y * n0)  # noqa: E731
        C, B = [h, z, *frame(qx, qy)], [h, z, *frame(gqx, gqy)]
        f, n, t, sa, _ = _edge_flux(self.order, C, B, list(C), list(B))
        return f, n * n0 - t * n1, n * n1 + t * n0, sa * n0, sa * n1

    def step(self, fixed_dt=None):
        dt, V = self.dt, self.valid
        h, z, qx, qy = self.h, self.z, self.qx, self.qy
        sh = lambda a, dy, dx: torch.roll(a, (-dy, -dx), (0, 1))  # noqa: E731
        dh, dqx, dqy = torch.zeros_like(h), torch.zeros_like(h), torch.zeros_like(h)
        for axis in (0, 1):
            # plus side: the cell to the east, or to the north (the row above)
            dy, dx = ((0, 1), (-1, 0))[axis]
            cells = (h, z, qx, qy) if axis == 0 else (h, z, qy, -qx)
            at = lambda k: [sh(a, k * dy, k * dx) for a in cells]  # noqa: E731
            both = V & sh(V, dy, dx)
            out = _faces(self.order, list(cells), at(1), at(-1), at(2), sh(V, -dy, -dx),
                         sh(V, 2 * dy, 2 * dx))
            f, n, t, sa, sb = [torch.where(both, x, torch.zeros_like(x)) for x in out]
            back = lambda a: sh(a, -dy, -dx)  # noqa: E731
            dh += back(f) - f
            if axis == 0:
                dqx += back(n + sb) - (n + sa)
                dqy += back(t) - t
            else:
                dqx += -back(t) + t
                dqy += back(n + sb) - (n + sa)
        for edge in self.edges:
            rr, cc = edge[2], edge[3]
            f, fx, fy, sx, sy = self._ghosts(*edge)
            dh[rr, cc] -= f
            dqx[rr, cc] -= fx + sx
            dqy[rr, cc] -= fy + sy
        if self.t == 0.0:
            active = V
        else:
            wet = self.counts & (h > HS)
            active = V & ((h > HS) | sh(wet, 0, 1) | sh(wet, 0, -1) | sh(wet, 1, 0) |
                          sh(wet, -1, 0))
        r = active.double() * (dt / self.dx)
        hu = dh * r + self._rain() * dt
        if self.cum is not None:
            a = self.cum + dt * self.soil["ks"]
            F1 = 0.5 * (a + (a * a + 4.0 * dt * self.soil["ks"] * (self.soil["psi"] + h) *
                             self.soil["dtheta"]).sqrt())
            dF = torch.where(active, torch.minimum(h, F1 - self.cum), 0.0)
            self.cum = self.cum + dF
            hu = hu - dF
        h2 = torch.where(V, h + hu, 0.0)
        wet = V & ~(h2 < HS)
        hw = torch.where(wet, h2, 1.0)
        x2, y2 = qx + dqx * r, qy + dqy * r
        a = dt * G * self.n * self.n * hw ** (-1.0 / 3.0) / (hw * hw)
        fct = 2.0 / (1.0 + (1.0 + 4.0 * a * (x2 * x2 + y2 * y2).sqrt()).sqrt())
        lim = 5.0 * hw * (hw * G).sqrt()

        def drag(q):
            temp = q * fct
            over = 2.0 * temp - q
            over = torch.where(over * temp <= 0.0, 0.0, over)
            q = torch.where(q.abs() > 1.0e-10, torch.where(temp.abs() > lim, over, temp), q)
            return torch.where(wet, q, 0.0)

        self.h, self.qx, self.qy = h2, drag(x2), drag(y2)
        self.h_max = torch.maximum(self.h_max, h2)
        # the scheme takes this root in single precision (correctly rounded by way of double)
        celerity = (G * hw).float().double().sqrt().float().double()
        speed = celerity + torch.maximum(self.qx.abs(), self.qy.abs()) / hw
        cand = torch.where(V & (h2 > HS), self.cfl * self.dx / speed, 60.0)
        nxt = min(float(cand.min()), 10.0 * dt)
        self.dt = nxt if fixed_dt is None else fixed_dt
        self.t += self.dt

    def raster(self, x):
        return x[1:-1, 1:-1]

    def state(self):
        out = {"h": self.raster(self.h), "qx": self.raster(self.qx), "qy": self.raster(self.qy),
               "h_max": self.raster(self.h_max)}
        if self.cum is not None:
            out["cum"] = self.raster(self.cum)
        return out


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    if kind == "ensemble":
        out = []
        for d in _members(case, seed):
            s = _Dense(d, 2)
            for _ in range(steps):
                s.step()
            out.append(s.state())
        return out
    d = _inputs(case, seed)
    if kind == "gauges":
        s = _Dense(d, 2, [1.2 * n for n in d["manning"]], 1.1)
        rows = torch.as_tensor(d["gauge_rows"], device=s.dev)
        cols = torch.as_tensor(d["gauge_cols"], device=s.dev)
        samples = []
        for k in range(1, steps + 1):
            s.step(fixed_dt=d["dt0"])
            if k % case["every"] == 0:
                samples.append(s.raster(s.h)[rows, cols])
        samples = torch.stack(samples)
        obs = torch.as_tensor(d["obs"], device=s.dev)
        # the gradients have no plain 64-bit counterpart here: the discrete adjoint is the
        # library's own
        return {"samples": samples, "loss": ((samples - obs) ** 2).sum(), "grad": None,
                "initial": {"h": None, "qx": None, "qy": None}}
    s = _Dense(d, case.get("order", 1 if kind == "coupled" else 2))
    if kind == "host":  # every step starts from the host's input buffers
        first = (s.h, s.qx, s.qy)
        for _ in range(steps):
            s.h, s.qx, s.qy = first
            s.step()
        v = s.valid
        return [s.h[v], s.qx[v], s.qy[v]]
    for _ in range(steps):
        s.step()
    if kind == "godunov":
        v = s.valid
        return {"h": s.h[v], "qx": s.qx[v], "qy": s.qy[v], "wl": (s.h + s.z)[v],
                "h_max": s.h_max[v]}
    out = [s.state()]
    if kind == "coupled":
        rr, cc = (torch.as_tensor(a, device=s.dev) for a in _agents(case, seed))
        h, qx, qy = (s.raster(x)[rr, cc] for x in (s.h, s.qx, s.qy))
        wet = h > HS
        out.append((h, torch.where(wet, qx / h, 0.0), torch.where(wet, qy / h, 0.0)))
    return out
