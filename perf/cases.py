"""The work that a user of this framework has it do, as cases to be timed and compared.

  listed()             the named cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  the simulation (or ensemble, adjoint, terrain document) a program holds before the call
  run(state)           one pass through the public entry points, and its outputs
  work(case)           bytes and operations a pass cannot do without
  exact(case, seed)    what run() returns, from plain torch in 64 bits

The kinds of case and what each stands for in use:

  rig        a verification rig: a small lake stepped one call at a time with dt = maxDt(), the
             diagnostics read at the end (the reference's suites, examples, teaching models)
  frame      an interactive window: a few step() calls, then the map panel as RGBA bytes on the host
  loop       a production run on the device: a scenario is loaded, advanced by run(n), and its
             state handed on in device memory; every boundary kind, limiter, friction form and
             wet/dry mix of the configurations, plain and odd sizes, up to 2048 x 2048
  globe      the same on the latitude-longitude grid with land, rotation and a tide at both edges
  diag       monitoring of a large run: volume, energy, largest speed and deviation, finiteness, maxDt
  globeview  one frame of the globe view of a spherical run, RGBA bytes and statistics on the host
  ensemble   many uneven basins with their own tides advanced together
  adjoint    one gauge-misfit gradient (forward and backward) for the bed and the Manning field
  import     a terrain document parsed, put on the device and asked for its first time step
"""
import base64
import ctypes
import math

import numpy as np
import torch

from __graft_entry__ import load_package

swe = load_package()
from water_simulator_b200 import workloads  # noqa: E402
from water_simulator_b200._lib import FIELD, check  # noqa: E402

G = 9.80665
OMEGA = 7.292115e-5
R_EARTH = 6371e3
STATE = ("h", "hu", "hv")


def listed():
    return [
        # the verification suites' 200 x 4 lake (walls W/E, periodic S/N): call latency and nothing else
        {"name": "rig_200x4", "kind": "rig", "nx": 200, "ny": 4, "steps": 20},
        # a teaching-size window redrawn after every 4 steps
        {"name": "frame_160x96", "kind": "frame", "nx": 160, "ny": 96, "steps": 4},
        # the plain configuration: bump and roughness, dam break, walls, Manning 0.025
        {"name": "dam_256", "kind": "loop", "bed": "bump", "nx": 256, "ny": 256, "steps": 100, "limiter": "mc",
         "sides": "walls", "friction": "scalar"},
        # an odd grid off the tuned path: minmod, per-cell Manning, open west and periodic south/north
        {"name": "channel_777x501", "kind": "loop", "bed": "bump", "nx": 777, "ny": 501, "steps": 128,
         "limiter": "minmod", "sides": "open", "friction": "field"},
        # every cell wet at the largest size: a lake or ocean basin in full motion
        {"name": "allwet_2048", "kind": "loop", "bed": "bump", "nx": 2048, "ny": 2048, "steps": 128, "limiter": "mc",
         "sides": "walls", "friction": "scalar"},
        # the flooding configuration: dam break over a beach, mostly dry land, Flather west
        {"name": "beach_2048", "kind": "loop", "bed": "beach", "nx": 2048, "ny": 2048, "steps": 128, "limiter": "mc",
         "sides": "flather", "friction": "scalar"},
        # the spherical configuration: 0.25 degrees, 30 % land, M2 tide at both edges
        {"name": "globe_1440x720", "kind": "globe", "nx": 1440, "ny": 720, "steps": 128},
        # monitoring between the chunks of a large run
        {"name": "diag_1536x1024", "kind": "diag", "nx": 1536, "ny": 1024},
        # the globe view at 900 pixels over a half-degree run
        {"name": "globeview_900", "kind": "globeview", "nx": 720, "ny": 360, "size": 900},
        # a share of the 256-basin ensemble configuration
        {"name": "ensemble_48", "kind": "ensemble", "basins": 48, "steps": 8},
        # one gradient, checkpoints every 45 steps as in the adjoint configuration
        {"name": "adjoint_512x384", "kind": "adjoint", "nx": 512, "ny": 384, "steps": 60, "gauges": 32},
        # a 50 m terrain export with its Manning layer
        {"name": "import_400x300", "kind": "import", "nx": 400, "ny": 300},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rig", "frame", "loop", "loop", "loop", "loop", "globe", "diag", "globeview", "ensemble",
                       "adjoint", "import"])
    if kind == "rig":
        return {"kind": kind, "nx": _log(rng, 16, 400), "ny": _log(rng, 4, 64), "steps": rng.randint(8, 32)}
    if kind == "frame":
        return {"kind": kind, "nx": _log(rng, 48, 512), "ny": _log(rng, 32, 384), "steps": rng.randint(1, 8)}
    if kind == "loop":
        bed = rng.choice(["bump", "bump", "beach"])
        lo = 64 if bed == "bump" else 384
        nx, ny = _log(rng, lo, 1700), _log(rng, lo, 1700)
        return {"kind": kind, "bed": bed, "nx": nx, "ny": ny, "steps": rng.choice([20, 32, 77, 128]),
                "limiter": rng.choice(["mc", "mc", "minmod"]),
                "sides": "flather" if bed == "beach" else rng.choice(["walls", "open"]),
                "friction": rng.choice(["scalar", "scalar", "field"])}
    if kind == "globe":
        nx = 2 * _log(rng, 90, 720)
        return {"kind": kind, "nx": nx, "ny": nx // 2, "steps": rng.choice([32, 77, 128])}
    if kind == "diag":
        return {"kind": kind, "nx": _log(rng, 64, 1900), "ny": _log(rng, 64, 1500)}
    if kind == "globeview":
        nx = 2 * _log(rng, 60, 720)
        return {"kind": kind, "nx": nx, "ny": nx // 2, "size": rng.randint(200, 1100)}
    if kind == "ensemble":
        return {"kind": kind, "basins": rng.randint(4, 64), "steps": rng.randint(2, 12)}
    if kind == "adjoint":
        return {"kind": kind, "nx": _log(rng, 64, 600), "ny": _log(rng, 64, 400), "steps": rng.randint(10, 90),
                "gauges": rng.randint(1, 48)}
    return {"kind": kind, "nx": _log(rng, 64, 600), "ny": _log(rng, 48, 450)}


# ---- inputs ------------------------------------------------------------------
def _loop_inputs(case, seed):
    """b, eta0, dx and the Manning argument of a loop case, over the padded grid."""
    nx, ny = case["nx"], case["ny"]
    if case["bed"] == "beach":
        b, h = workloads.beach_dam_break(nx, ny, 2.0, seed=seed, x_dam=min(500.0, 0.3 * nx * 2.0))
        eta, dx, manning = b + h, 2.0, 0.03
    else:
        b, eta = workloads.bump_dam_break(nx, ny, 5.0, seed=seed)
        if nx * ny > 1 << 20 or case["sides"] == "open":      # every cell wet
            X = np.arange(nx + 4)[None, :]
            eta = np.broadcast_to(np.where(X < nx // 2, 3.0, 2.5), b.shape).copy()
            b = np.minimum(b, 1.7)
        dx, manning = 5.0, 0.025
    if case["friction"] == "field":
        manning = workloads.uniform_noise(seed + 77, b.shape, 0.015, 0.04)
    return b, eta, dx, manning


def _lake_inputs(case, seed):
    """The lake rig: 2 m over a smooth bump with seeded roughness, a released 0.2 m hump to set it moving."""
    nx, ny, dx = case["nx"], case["ny"], 5.0
    X, Y = np.meshgrid((np.arange(nx + 4) - 1.5) * dx, (np.arange(ny + 4) - 1.5) * dx)
    L = nx * dx
    b = 0.8 * np.exp(-((X - 0.5 * L) / (0.12 * L)) ** 2) + workloads.uniform_noise(seed, X.shape, -0.1, 0.1)
    eta = 2.0 + 0.2 * np.exp(-((X - 0.25 * L) / (0.08 * L)) ** 2)
    return b, eta, dx


def _globe_inputs(case, seed):
    return workloads.globe_tide(case["nx"], case["ny"], seed=seed)


def _ensemble_sizes(n):
    """The sizes of the ensemble configuration's first n basins, nx ~ U[64, 1024] and ny ~ U[64, 512]."""
    rng = np.random.default_rng(4)
    return [(int(rng.integers(64, 1025)), int(rng.integers(64, 513))) for _ in range(n)]


def _ensemble_inputs(case, seed):
    """Basins as workloads.ensemble() describes them, their beds, friction and tides made from the seed."""
    rng = np.random.default_rng(seed)
    out = []
    for q, (nx, ny) in enumerate(_ensemble_sizes(case["basins"])):
        period = 3600 * rng.uniform(2.0, 14.0)
        out.append({"nx": nx, "ny": ny, "dx": 5.0, "b": workloads.bump_bed(nx, ny, 5.0, seed=1000 * seed + q),
                    "eta0": 2.0, "manning": float(rng.uniform(0.015, 0.04)),
                    "tide": {"msl": 2.0, "amp": [0.5], "omega": [2 * math.pi / period], "phase_deg": [0.0]}})
    return out


def _diag_inputs(case, seed):
    """A state in motion: depths around 2 m over roughness, a fifth of it dry land, velocities of some 0.5 m/s."""
    shape = (case["ny"] + 4, case["nx"] + 4)
    b = workloads.uniform_noise(seed, shape, -0.5, 0.5)
    h = workloads.uniform_noise(seed + 1, shape, 1.0, 3.0)
    h[:, : shape[1] // 5] = 0.0
    hu = h * workloads.uniform_noise(seed + 2, shape, -0.5, 0.5)
    hv = h * workloads.uniform_noise(seed + 3, shape, -0.5, 0.5)
    return b, h, hu, hv


def _terrain_doc(case, seed):
    """A gridlands-terrain v1 document of a sloping map: sea in the south, dry land with one lake, Manning classes."""
    W, H = case["nx"], case["ny"]
    r, c = np.arange(H)[:, None] / H, np.arange(W)[None, :] / W
    bed = 60 - 110 * r ** 1.5 + 6 * np.sin(18 * c + seed % 7) + workloads.uniform_noise(seed, (H, W), -0.5, 0.5)
    lake = (r - 0.3) ** 2 + (c - 0.4) ** 2 < 0.01
    bed = np.where(lake, bed - 8, bed).astype(np.float32)
    surf = np.where(bed < 0, np.float32(0), np.where(lake, np.maximum(bed, np.float32(40)), bed)).astype(np.float32)
    n = np.where(surf > bed, 0.02, np.where(bed < 20, 0.035, 0.1)).astype(np.float32)

    def layer(a):
        return {"encoding": "b64f32le", "data": base64.b64encode(a.astype("<f4").tobytes()).decode("ascii")}

    doc = {"format": "gridlands-terrain", "version": 1,
           "grid": {"width": W, "height": H, "cellMeters": 50.0, "rowOrder": "north-first"},
           "layers": {"bedM": layer(bed), "surfaceM": layer(surf), "manningN": layer(n)},
           "stats": {"suggestedManningScalar": 0.035}, "meta": {"tool": "gridlands", "seed": int(seed)}}
    return doc, bed, surf, n


def _open_sides(sim):
    sim.boundaries.west = swe.outflow
    sim.boundaries.south = swe.periodic
    sim.boundaries.north = swe.periodic


def _globe_sim(case, seed):
    g = _globe_inputs(case, seed)
    sim = swe.ShallowWater(nx=case["nx"], ny=case["ny"], bed=g["b"], eta0=g["eta0"], manning=0.025,
                           sphere={"lat0": g["lat0"], "lat1": g["lat1"], "omega": OMEGA})
    tide = swe.Tide({"M2": [1.0, 30.0]}).signal()
    sim.boundaries.south = swe.flather(tide)
    sim.boundaries.north = swe.flather(tide)
    return sim


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind == "rig":
        b, eta, dx = _lake_inputs(case, seed)
        st["sim"] = swe.ShallowWater(nx=case["nx"], ny=case["ny"], dx=dx, bed=b, eta0=eta, manning=0)
        st["sim"].boundaries = {"south": swe.periodic, "north": swe.periodic}
    elif kind == "frame":
        b, eta, dx = _lake_inputs(case, seed)
        st["sim"] = swe.ShallowWater(nx=case["nx"], ny=case["ny"], dx=dx, bed=b, eta0=eta, manning=0.025)
    elif kind == "loop":
        b, eta, dx, n = _loop_inputs(case, seed)
        sim = swe.ShallowWater(nx=case["nx"], ny=case["ny"], dx=dx, bed=b, eta0=eta, limiter=case["limiter"],
                               manning=n if np.isscalar(n) else 0.025)
        if not np.isscalar(n):
            sim.setManningField(n)
        if case["sides"] == "flather":
            sim.boundaries.west = swe.flather(swe.Tide({}, msl=0.0).signal())
        elif case["sides"] == "open":
            _open_sides(sim)
        st["sim"] = sim
    elif kind == "globe":
        st["sim"] = _globe_sim(case, seed)
    elif kind == "diag":
        b, h, hu, hv = _diag_inputs(case, seed)
        sim = swe.ShallowWater(nx=case["nx"], ny=case["ny"], dx=5.0, bed=b, eta0=b + h)
        sim.h, sim.hu, sim.hv = h, hu, hv
        sim.maxDt()                                   # the fields are on the device from here on
        st["sim"] = sim
    elif kind == "globeview":
        sim = _globe_sim(case, seed)
        sim.run(8)
        cam = swe.globeCamera(case["size"], tiltDeg=22)
        st.update(sim=sim, lut=swe.buildGlobeLut(cam, sim), frame=0,
                  rgba=np.empty(4 * case["size"] ** 2, dtype=np.uint8))
    elif kind == "ensemble":
        st["ens"] = swe.Ensemble(_ensemble_inputs(case, seed))
    elif kind == "adjoint":
        a = workloads.adjoint_case(case["nx"], case["ny"], n_gauges=case["gauges"], seed=seed)
        obs = 2.0 + 0.01 * np.random.default_rng(seed).standard_normal((case["steps"], case["gauges"]))
        adj = swe.MisfitAdjoint(case["nx"], case["ny"], a["dx"], a["b"], a["eta0"], manning_field=a["n"],
                                gauges=a["gauges"], steps=case["steps"])
        adj.set_observations(obs)
        st["adj"] = adj
    else:
        st["doc"] = _terrain_doc(case, seed)[0]
    if kind in ("loop", "globe"):                     # the scenario a pass starts from, and where its result goes
        st["start"] = {f: torch.from_numpy(np.array(st["sim"].field(f))).cuda() for f in STATE}
        st["out"] = {f: torch.empty_like(st["start"][f]) for f in STATE}
    return st


def _load_state(sim, src):
    for f in STATE:
        check(sim._lib.swe_set_rows_async(sim._h, FIELD[f], 0, sim.H, ctypes.c_void_p(src[f].data_ptr())))


def _hand_on(sim, dst):
    for f in STATE:
        check(sim._lib.swe_get_rows_async(sim._h, FIELD[f], 0, sim.H, ctypes.c_void_p(dst[f].data_ptr())))
    return dst


def _watched(n):
    return sorted({0, n // 2, n - 1})


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "rig":
        sim = st["sim"]
        taken = [sim.step(sim.maxDt()) for _ in range(case["steps"])]
        return {"dt": np.array(taken), "h": sim.field("h"), "hu": sim.field("hu"), "hv": sim.field("hv"),
                "volume": sim.volume(), "dev": sim.maxSurfaceDeviation(2.0), "speed": sim.maxSpeed()}
    if kind == "frame":
        sim = st["sim"]
        taken = [sim.step() for _ in range(case["steps"])]
        return {"dt": np.array(taken), "rgba": swe.renderMap(sim, msl=2.0, scale=0.3), "h": sim.field("h")}
    if kind in ("loop", "globe"):
        sim = st["sim"]
        _load_state(sim, st["start"])
        sim.run(case["steps"])
        return _hand_on(sim, st["out"])
    if kind == "diag":
        sim = st["sim"]
        return {"volume": sim.volume(), "energy": sim.energy(), "dev": sim.maxSurfaceDeviation(2.0),
                "speed": sim.maxSpeed(), "finite": sim.finite(), "dt": sim.maxDt()}
    if kind == "globeview":
        st["frame"] += 1
        s = swe.renderGlobe(st["rgba"], st["sim"], st["lut"], rotDeg=7.5 * st["frame"], scale=0.5)
        return {"rgba": st["rgba"], "wet": s["wet"], "dry": s["dry"], "sat": s["sat"], "etaMin": s["etaMin"],
                "etaMax": s["etaMax"]}
    if kind == "ensemble":
        ens = st["ens"]
        ens.run(case["steps"])
        ens.synchronize()
        # the basins a program watches while the ensemble runs on
        return [{f: ens.field(q, f) for f in STATE} | {"t": ens.t(q)} for q in _watched(ens.n)]
    if kind == "adjoint":
        J, eta = st["adj"].forward()
        gb, gn = st["adj"].backward()
        return {"J": J, "eta": eta, "gb": gb, "gn": gn}
    t = swe.gridlandsTerrain(st["doc"])
    sim = swe.ShallowWater.fromGridlands(t, manningField=True)
    out = {"dt": sim.maxDt(), "b": sim.field("b"), "h": sim.field("h"), "n": sim.manningField}
    sim.close()
    return out


def work(case):
    """Per cell-update 136 bytes (stage 1 reads b and the state and writes it, stage 2 reads it all twice over) and
    some 1200 operations; the other paths read each input and write each output once."""
    kind = case["kind"]
    if kind == "ensemble":
        cells = sum(nx * ny for nx, ny in _ensemble_sizes(case["basins"]))
        return {"bytes": 136.0 * cells * case["steps"], "flops": 1200.0 * cells * case["steps"]}
    cells = case["nx"] * case["ny"]
    if kind in ("rig", "frame", "loop", "globe"):
        return {"bytes": 136.0 * cells * case["steps"], "flops": 1200.0 * cells * case["steps"]}
    if kind == "adjoint":                             # two forwards and a reverse that reads and writes as much again
        return {"bytes": 4 * 136.0 * cells * case["steps"], "flops": 4800.0 * cells * case["steps"]}
    if kind == "diag":
        return {"bytes": 32.0 * cells, "flops": 60.0 * cells}
    if kind == "globeview":
        return {"bytes": 36.0 * case["size"] ** 2, "flops": 20.0 * case["size"] ** 2}
    return {"bytes": (16.0 + 40.0) * cells, "flops": 30.0 * cells}


# ---- the step in plain torch, 64 bits ------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _metric(ny, dx=None, nx=None, lat0=None, lat1=None, omega=0.0):
    """The metric rows (src/geometry.mjs:163-299) as columns that broadcast over a padded grid."""
    H = ny + 4
    if dx is not None:
        one = np.ones(H)
        m = {"dx": dx * one, "dyN": dx * one, "dyS": dx * one, "dyC": dx * one, "bed": dx * one, "geo": 0 * one,
             "f": 0 * one, "tan": 0 * one}
        R, sph = math.inf, False
    else:
        R, sph = R_EARTH, True
        dlam, p0, p1 = 2 * math.pi / nx, math.radians(lat0), math.radians(lat1)
        dphi = (p1 - p0) / ny
        j = np.arange(H) - 2
        pS = np.clip(p0 + j * dphi, -math.pi / 2, math.pi / 2)
        pN = np.clip(p0 + (j + 1) * dphi, -math.pi / 2, math.pi / 2)
        pC = 0.5 * (pS + pN)
        lyS, lyN, lx = R * dlam * np.cos(pS), R * dlam * np.cos(pN), R * dphi
        A = 2 * R * R * dlam * np.cos(pC) * np.sin(0.5 * (pN - pS))
        m = {"dx": A / lx, "dyN": A / lyN, "dyS": A / lyS, "bed": 2 * A / (lyN + lyS), "geo": (lyN - lyS) / (4 * A),
             "f": 2 * omega * np.sin(pC), "tan": np.tan(pC)}
        m["dyC"] = np.minimum(np.minimum(m["dyN"], m["dyS"]), R * dphi)
    m = {k: torch.tensor(v, dtype=torch.float64, device=_device())[:, None] for k, v in m.items()}
    return m | {"R": R, "sph": sph}


class _Plain:
    """ShallowWater's step over whole arrays: the formulas of src/swe.mjs, torch operations in 64 bits."""

    def __init__(self, b, h, metric, sides, manning, limiter="mc", flather=None, dry=1e-3, cfl=0.45):
        def t(a):
            return torch.tensor(np.asarray(a), dtype=torch.float64, device=_device())
        self.b, self.h = t(b), t(h)
        self.hu, self.hv = torch.zeros_like(self.h), torch.zeros_like(self.h)
        self.m, self.sides, self.limiter, self.flather = metric, sides, limiter, flather or {}
        self.n = None if np.isscalar(manning) and manning == 0 else (manning if np.isscalar(manning) else t(manning))
        self.dry, self.cfl, self.eps4, self.t = dry, cfl, dry ** 4, 0.0

    def vel(self, q, h):
        h4 = h * h * h * h
        return math.sqrt(2) * h * q / torch.sqrt(h4 + torch.clamp(h4, min=self.eps4))

    def ghosts(self, h, hu, hv):
        for side, kind in (("west", self.sides[0]), ("east", self.sides[1]), ("south", self.sides[2]),
                           ("north", self.sides[3])):
            ax = 1 if side in ("west", "east") else 0
            n = self.b.shape[ax] - 4
            for g in range(2):
                at = 1 - g if side in ("west", "south") else n + 2 + g
                near = 2 if side in ("west", "south") else n + 1
                src = {"reflect": 3 - at if near == 2 else 2 * n + 3 - at, "periodic": at + n if near == 2 else at - n,
                       "outflow": near, "flather": near}[kind]
                new = [f.select(ax, src).clone() for f in (self.b, h, hu, hv)]
                if ax == 0 and kind != "periodic":      # corners come from the nearest interior column
                    for v in new:
                        v[:2], v[-2:] = v[2].clone(), v[-3].clone()
                norm = 2 if ax == 1 else 3
                if kind == "reflect":
                    new[norm] = -new[norm]
                elif kind == "flather":
                    bb, hh = new[0], new[1]
                    e0, u0 = self.flather[side](self.t), 0.0
                    wet = hh > self.dry
                    hs = torch.where(wet, hh, torch.ones_like(hh))
                    r, s = torch.sqrt(G / hs), 1.0 if near == 2 else -1.0
                    rin, rout = u0 + s * e0 * r, self.vel(new[norm], hs) - s * (bb + hs) * r
                    hg = torch.where(wet, torch.clamp(s * (rin - rout) / (2 * r) - bb, min=0),
                                     torch.clamp(e0 - bb, min=0))
                    new[1] = hg
                    new[norm] = torch.where(wet, hg * 0.5 * (rin + rout), torch.zeros_like(hg))
                    new[5 - norm] = torch.where(wet, new[5 - norm], torch.zeros_like(hg))
                for f, v in zip((self.b, h, hu, hv), new):
                    f.select(ax, at).copy_(v)

    def lim(self, a, c):
        z = torch.zeros_like(a)
        if self.limiter == "minmod":
            return torch.where((a > 0) & (c > 0), torch.minimum(a, c),
                               torch.where((a < 0) & (c < 0), torch.maximum(a, c), z))
        s = torch.minimum(torch.minimum((0.5 * (a + c)).abs(), 2 * a.abs()), 2 * c.abs())
        return torch.where(a * c > 0, torch.where(a > 0, s, -s), z)

    def slopes(self, h, u, v, ax):
        out = [torch.zeros_like(h) for _ in range(4)]
        n = h.shape[ax]
        lo, mid, hi = (lambda f, k=k: f.narrow(ax, k, n - 2) for k in range(3))
        wet = (lo(h) > self.dry) & (mid(h) > self.dry) & (hi(h) > self.dry)
        for o, f in zip(out, (self.b + h, self.b, u, v)):
            mid(o).copy_(torch.where(wet, self.lim(mid(f) - lo(f), hi(f) - mid(f)), torch.zeros_like(mid(h))))
        edge = 1 - ax                                   # no slopes in the outermost ring
        for o in out:
            o.select(edge, 0).zero_()
            o.select(edge, h.shape[edge] - 1).zero_()
        return out

    def faces(self, h, nv, tv, s, ax):
        """Mass, normal + left and right pressure, transverse flux between each cell and the next along ax."""
        n = h.shape[ax] - 1
        L, R = (lambda f: f.narrow(ax, 0, n)), (lambda f: f.narrow(ax, 1, n))
        sE, sB, sN, sT = s
        eL, eR = L(self.b) + L(h) + 0.5 * L(sE), R(self.b) + R(h) - 0.5 * R(sE)
        bL, bR = L(self.b) + 0.5 * L(sB), R(self.b) - 0.5 * R(sB)
        hLf, hRf = torch.clamp(eL - bL, min=0), torch.clamp(eR - bR, min=0)
        top = torch.maximum(bL, bR)
        hL, hR = torch.clamp(eL - top, min=0), torch.clamp(eR - top, min=0)
        wL, wR = hL > self.dry, hR > self.dry
        z, one = torch.zeros_like(hL), torch.ones_like(hL)
        quL, quR = hL * (L(nv) + 0.5 * L(sN)), hR * (R(nv) - 0.5 * R(sN))
        qvL, qvR = hL * (L(tv) + 0.5 * L(sT)), hR * (R(tv) - 0.5 * R(sT))
        sl, sr = torch.where(wL, hL, one), torch.where(wR, hR, one)
        uL, vL = torch.where(wL, quL / sl, z), torch.where(wL, qvL / sl, z)
        uR, vR = torch.where(wR, quR / sr, z), torch.where(wR, qvR / sr, z)
        cL, cR = torch.sqrt(G * hL), torch.sqrt(G * hR)
        a = (cL + cR) / 2 + (uL - uR) / 4
        hs = a * a / G
        gL = torch.where(hs > hL, torch.sqrt(0.5 * (hs + hL) * hs / (sl * sl)), one)
        gR = torch.where(hs > hR, torch.sqrt(0.5 * (hs + hR) * hs / (sr * sr)), one)
        SL = torch.where(~wL, uR - 2 * cR, torch.where(~wR, uL - cL, uL - cL * gL))
        SR = torch.where(~wL, uR + cR, torch.where(~wR, uL + 2 * cL, uR + cR * gR))
        num = SL * hR * (uR - SR) - SR * hL * (uL - SL)
        den = hR * (uR - SR) - hL * (uL - SL)
        big = den.abs() > 1e-30
        SM = torch.where(big, num / torch.where(big, den, one), 0.5 * (SL + SR))
        pl, pr = quL * uL + 0.5 * G * hL * hL, quR * uR + 0.5 * G * hR * hR
        dS = torch.where(SR > SL, SR - SL, one)
        M = (SR * quL - SL * quR + SL * SR * (hR - hL)) / dS
        N = (SR * pl - SL * pr + SL * SR * (quR - quL)) / dS
        T = M * torch.where(SM >= 0, vL, vR)
        left, right, dead = SL >= 0, SR <= 0, ~wL & ~wR
        M = torch.where(dead, z, torch.where(left, quL, torch.where(right, quR, M)))
        N = torch.where(dead, z, torch.where(left, pl, torch.where(right, pr, N)))
        T = torch.where(dead, z, torch.where(left, qvL * uL, torch.where(right, qvR * uR, T)))
        return M, N + 0.5 * G * (hLf * hLf - hL * hL), N + 0.5 * G * (hRf * hRf - hR * hR), T

    def residual(self, h, hu, hv, dt):
        """d(h, hu, hv)/dt of the interior cells; every array below is the padded grid's, faces by their lower cell."""
        m = self.m
        u, v = self.vel(hu, h), self.vel(hv, h)
        sx, sy = self.slopes(h, u, v, 1), self.slopes(h, u, v, 0)
        fx = [torch.nn.functional.pad(f, (0, 1)) for f in self.faces(h, u, v, sx, 1)]
        fy = [torch.nn.functional.pad(f, (0, 0, 0, 1)) for f in self.faces(h, v, u, (sy[0], sy[1], sy[3], sy[2]), 0)]
        for f in fx:
            f[:2], f[-2:], f[:, 0], f[:, -2:] = 0, 0, 0, 0
        for f in fy:
            f[:, :2], f[:, -2:], f[0], f[-2:] = 0, 0, 0, 0
        W, S = (lambda f: torch.roll(f, 1, 1)), (lambda f: torch.roll(f, 1, 0))
        out = (torch.clamp(fx[0], min=0) - torch.clamp(W(fx[0]), max=0)) / m["dx"] \
            + torch.clamp(fy[0], min=0) / m["dyN"] - torch.clamp(S(fy[0]), max=0) / m["dyS"]
        over = out * dt > h
        th = torch.where(over, torch.where(h > 0, h / torch.where(over, out * dt, torch.ones_like(h)),
                                           torch.zeros_like(h)), torch.ones_like(h))
        tx = torch.where(fx[0] >= 0, th, torch.roll(th, -1, 1))
        ty = torch.where(fy[0] >= 0, th, torch.roll(th, -1, 0))
        ah = W(fx[0] * tx) / m["dx"] - fx[0] * tx / m["dx"] + S(fy[0] * ty) / m["dyS"] - fy[0] * ty / m["dyN"]
        au = W(fx[2] * tx) / m["dx"] - fx[1] * tx / m["dx"] + S(fy[3] * ty) / m["dyS"] - fy[3] * ty / m["dyN"]
        av = W(fx[3] * tx) / m["dx"] - fx[3] * tx / m["dx"] + S(fy[2] * ty) / m["dyS"] - fy[1] * ty / m["dyN"]

        def bed(sE, sB):
            P = torch.clamp(h + 0.5 * sE - 0.5 * sB, min=0)
            Q = torch.clamp(h - 0.5 * sE + 0.5 * sB, min=0)
            return -G * 0.5 * (P + Q) * sB, P * P + Q * Q
        bx, _ = bed(sx[0], sx[1])
        by, sq = bed(sy[0], sy[1])
        eu, ev = bx / m["dx"], by / m["bed"]
        if m["sph"]:
            fe = m["f"] + u * (m["tan"] / m["R"])
            eu, ev = eu + fe * hv, ev + m["geo"] * G * sq - fe * hu
        inner = torch.zeros_like(h)                     # the sources act on interior cells
        inner[2:-2, 2:-2] = 1
        return ah, au + inner * eu, av + inner * ev

    def clean(self, h, hu, hv):
        wet = torch.zeros_like(h, dtype=torch.bool)
        wet[2:-2, 2:-2] = True
        h = torch.where(wet & (h < 0), torch.zeros_like(h), h)
        kill = wet & (h <= self.dry)
        return h, torch.where(kill, torch.zeros_like(h), hu), torch.where(kill, torch.zeros_like(h), hv)

    def max_dt(self):
        h, hu, hv = (f[2:-2, 2:-2] for f in (self.h, self.hu, self.hv))
        c = torch.sqrt(G * torch.clamp(h, min=0))
        rate = (self.vel(hu, h).abs() + c) / self.m["dx"][2:-2] + (self.vel(hv, h).abs() + c) / self.m["dyC"][2:-2]
        return self.cfl / float(torch.where(h > self.dry, rate, torch.zeros_like(h)).max())

    def step(self, dt=None):
        dt = self.max_dt() if dt is None else dt
        h0, u0, v0 = self.h, self.hu, self.hv
        self.ghosts(h0, u0, v0)
        r = self.residual(h0, u0, v0, dt)
        h, hu, hv = self.clean(*(q + dt * a for q, a in zip((h0, u0, v0), r)))
        self.ghosts(h, hu, hv)
        r = self.residual(h, hu, hv, dt)
        new = [0.5 * (p + q + dt * a) for p, q, a in zip((h0, u0, v0), (h, hu, hv), r)]
        h, hu, hv = self.clean(*new)
        if self.n is not None:
            wet = h > self.dry
            hs = torch.where(wet, h, torch.ones_like(h))
            speed = torch.hypot(self.vel(hu, hs), self.vel(hv, hs))
            k = torch.where(wet & (speed >= 1e-14), 1 + dt * G * self.n * self.n * speed / hs ** (4 / 3),
                            torch.ones_like(h))
            k[:2], k[-2:], k[:, :2], k[:, -2:] = 1, 1, 1, 1
            hu, hv = hu / k, hv / k
        self.h, self.hu, self.hv, self.t = h, hu, hv, self.t + dt
        return dt


WALLS = ("reflect",) * 4


def _globe_plain(case, seed):
    g = _globe_inputs(case, seed)
    m = _metric(case["ny"], nx=case["nx"], lat0=g["lat0"], lat1=g["lat1"], omega=OMEGA)

    def tide(t):
        return math.cos(2 * math.pi / (12.4206012 * 3600) * t - 30.0 * math.pi / 180)
    return _Plain(g["b"], np.maximum(g["eta0"] - g["b"], 0), m, ("periodic", "periodic", "flather", "flather"), 0.025,
                  flather={"south": tide, "north": tide})


def exact(case, seed):
    kind = case["kind"]
    inner = (slice(2, -2), slice(2, -2))
    if kind in ("rig", "frame"):
        b, eta, dx = _lake_inputs(case, seed)
        sides = ("reflect", "reflect", "periodic", "periodic") if kind == "rig" else WALLS
        p = _Plain(b, np.maximum(eta - b, 0), _metric(case["ny"], dx=dx), sides, 0 if kind == "rig" else 0.025)
        taken = np.array([p.step() for _ in range(case["steps"])])
        if kind == "frame":
            return {"dt": taken, "rgba": None, "h": p.h.reshape(-1)}
        h = p.h[inner]
        speed = torch.hypot(p.vel(p.hu, p.h), p.vel(p.hv, p.h))[inner]
        return {"dt": taken, "h": p.h.reshape(-1), "hu": p.hu.reshape(-1), "hv": p.hv.reshape(-1),
                "volume": float(h.sum()) * dx * dx, "dev": float((p.b[inner] + h - 2.0).abs().max()),
                "speed": float(speed.max())}
    if kind in ("loop", "globe"):
        if kind == "globe":
            p = _globe_plain(case, seed)
        else:
            b, eta, dx, n = _loop_inputs(case, seed)
            sides = {"walls": WALLS, "open": ("outflow", "reflect", "periodic", "periodic"),
                     "flather": ("flather", "reflect", "reflect", "reflect")}[case["sides"]]
            p = _Plain(b, np.maximum(eta - b, 0), _metric(case["ny"], dx=dx), sides, n, case["limiter"],
                       {"west": lambda t: 0.0})
        for _ in range(case["steps"]):
            p.step()
        return {f: getattr(p, f).reshape(-1) for f in STATE}
    if kind == "diag":
        b, h, hu, hv = _diag_inputs(case, seed)
        p = _Plain(b, h, _metric(case["ny"], dx=5.0), WALLS, 0.025)
        p.hu, p.hv = (torch.tensor(a, dtype=torch.float64, device=_device()) for a in (hu, hv))
        hh, bb = p.h[inner], p.b[inner]
        u, v = p.vel(p.hu, p.h)[inner], p.vel(p.hv, p.h)[inner]
        wet = hh > p.dry
        z = torch.zeros_like(hh)
        e = torch.where(hh > 0, 0.5 * hh * (u * u + v * v) + 0.5 * G * hh * (hh + 2 * bb), z)
        return {"volume": float(hh.sum()) * 25.0, "energy": float(e.sum()) * 25.0,
                "dev": float(torch.where(wet, (bb + hh - 2.0).abs(), z).max()),
                "speed": float(torch.where(wet, torch.hypot(u, v), z).max()), "finite": True, "dt": p.max_dt()}
    if kind == "ensemble":
        out = []
        for q, bs in enumerate(_ensemble_inputs(case, seed)):
            if q not in _watched(case["basins"]):
                continue
            td = bs["tide"]

            def tide(t, td=td):
                return td["msl"] + td["amp"][0] * math.cos(td["omega"][0] * t)
            p = _Plain(bs["b"], np.maximum(bs["eta0"] - bs["b"], 0), _metric(bs["ny"], dx=bs["dx"]),
                       ("flather", "reflect", "reflect", "reflect"), bs["manning"], flather={"west": tide})
            for _ in range(case["steps"]):
                p.step()
            out.append({f: getattr(p, f).reshape(-1) for f in STATE} | {"t": p.t})
        return out
    if kind == "adjoint":
        a = workloads.adjoint_case(case["nx"], case["ny"], n_gauges=case["gauges"], seed=seed)
        obs = 2.0 + 0.01 * np.random.default_rng(seed).standard_normal((case["steps"], case["gauges"]))
        p = _Plain(a["b"], np.maximum(a["eta0"] - a["b"], 0), _metric(case["ny"], dx=a["dx"]), WALLS, a["n"])
        at = torch.tensor(a["gauges"].astype(np.int64), device=_device())
        eta = np.empty((case["steps"], case["gauges"]))
        for k in range(case["steps"]):
            p.step()
            eta[k] = (p.b + p.h).reshape(-1)[at].cpu().numpy()
        return {"J": float(((eta - obs) ** 2).sum()), "eta": eta, "gb": None, "gn": None}
    if kind == "import":
        _, bed, surf, n = _terrain_doc(case, seed)

        def grid(a):
            return np.pad(a[::-1].astype(np.float64), 2, mode="edge")
        b, h = grid(bed), np.maximum(grid(surf) - grid(bed), 0)
        p = _Plain(b, h, _metric(case["ny"], dx=50.0), WALLS, 0.035)
        return {"dt": p.max_dt(), "b": b.reshape(-1), "h": h.reshape(-1), "n": grid(n).reshape(-1)}
    return None
