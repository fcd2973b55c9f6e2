"""The work a user of this package has it do, as measurable cases.

A case is a dict of plain values; ``prepare`` builds what a program holds
before the call (a mesh's solver with its initial state), ``run`` is one pass
through the public entry points, ``exact`` the same pass in float64 torch.

Kinds of case:

* ``run``      -- ``SWESolverB200Resident.run`` of one mesh from its initial state, with
  output windows and the state read back: one scenario of a flood study.
* ``phases``   -- the same run cut into phases with their own inflow rates, each resumed
  where the last ended, as the workflow drives a solver.
* ``channel``  -- a river reach open at both ends (inflow above, normal depth below).
* ``batch``    -- ``BatchedSolver.run`` of one or more scenarios with their own clocks
  (rain on every cell, or an inflow hydrograph each).
* ``gradient`` -- ``GaugeCalibration``: the gauge misfit and its gradient with respect to
  Manning's n, the bed and the hydrograph's knots, one iteration of a calibration.

Meshes are Voronoi diagrams of random points (sizes as in the package's
scenarios: 8 thousand cells to over a million), regular quads or channel
grids. A large Voronoi mesh is a random patch continued by reflection, which
is the exact Voronoi diagram of the reflected points and takes a fraction of
the time of a diagram of them all. A mesh belongs to its case; beds, initial
states, roughness and inflows come from the seed.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from inundation_b200.adjoint import GaugeCalibration
from inundation_b200.backend import SWESolverB200Resident
from inundation_b200.batch import BatchedSolver, BatchMember
from inundation_b200.mesh.boundaries import select_boundary_edges
from inundation_b200.mesh.geometry import build_geometry, hilbert_reorder, with_bed
from inundation_b200.mesh.synthetic import channel_grid, fractal_dem, gaussian_bumps, quad_grid, voronoi_mesh
from inundation_b200.sources import Hydrograph

GRAVITY, DRY_TOL, FILM_DEPTHS, TICKS = 9.81, 1e-4, 4.0, 1 << 20
OPEN_NORMAL, OPEN_INFLOW = 2, 4
PATCH_CELLS = 9000
SPACING = 10.0  # metres between cell centres of the Voronoi meshes

_RUN = {"kind": "run", "mesh": "voronoi", "windows": 2, "dt_max": 1.0, "cfl": 0.8, "compensated": True, "clamp": False}


def listed() -> list[dict]:
    return [
        # a restart of a small model over a handful of fixed steps: nothing but latency
        {**_RUN, "name": "valley 2k, 8 steps", "mesh": "quad", "cells": 2048, "water": "dam", "radius": 0.2,
         "seconds": 2.0**-7, "dt_max": 2.0**-10, "windows": 1},
        # a small lake, everything wet, CFL 0.9: the smallest of the package's configurations
        {**_RUN, "name": "lake 8k", "cells": 8000, "water": "lake", "cfl": 0.9, "seconds": 120.0},
        # a reach open at both ends, as in the validation channels
        {"name": "open channel 6k", "kind": "channel", "cells": 300, "across": 20, "seconds": 600.0, "windows": 3},
        # inflows that change from phase to phase, each phase resumed: the workflow's loop
        {"name": "inflow phases 30k", "kind": "phases", "cells": 30_011, "phases": 3, "seconds": 20.0, "inflows": 7},
        # plain depth (no low word) with the clamp tally kept: the two options of the update
        {**_RUN, "name": "dam break 70k, plain depth", "cells": 70_000, "water": "dam", "radius": 0.12,
         "seconds": 30.0, "compensated": False, "clamp": True},
        # a flood that has spread over a fifth of its mesh: between a front and a full mesh
        {**_RUN, "name": "flood 260k", "cells": 260_000, "water": "dam", "radius": 0.27, "seconds": 24.0},
        # the benchmark's dam break: a front in a mostly dry million cells
        {**_RUN, "name": "dam break 1m", "cells": 1_000_000, "water": "dam", "radius": 0.05, "seconds": 60.0},
        # every cell wet: a tidal flat or a filled basin
        {**_RUN, "name": "full basin 600k", "cells": 600_000, "water": "wet", "seconds": 10.0, "windows": 1},
        # rain on every cell and one inflow on ground already wetted
        {"name": "rain 1.2m", "kind": "batch", "members": 1, "cells": 1_200_000, "spread": 1.0, "rain": True,
         "seconds": 60.0},
        # an ensemble: meshes of uneven sizes, each with its own inflow and clock
        {"name": "ensemble of 16", "kind": "batch", "members": 16, "cells": 36_000, "spread": 3.0, "rain": False,
         "seconds": 30.0},
        # one iteration of a calibration, small and long enough for several checkpoints
        {"name": "gradient 30k", "kind": "gradient", "cells": 30_000, "steps": 100, "every": 40, "gauges": 60, "knots": 16},
        # the same at the size of the package's calibration scenario
        {"name": "gradient 250k", "kind": "gradient", "cells": 250_000, "steps": 200, "every": 50, "gauges": 200, "knots": 32},
    ]


def _log(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng) -> dict:
    """One more case of the listed ranges."""
    kind = rng.choice(["run", "run", "run", "run", "phases", "channel", "batch", "batch", "gradient"])
    if kind == "run":
        water = rng.choice(["lake", "dam", "dam", "wet"])
        cells = int(_log(rng, 2000, 1_000_000 if water == "dam" else 600_000))
        # the larger the mesh, the shorter the drawn run, so that no draw outgrows the listed ones
        steps = _log(rng, 8, min(600.0, 60e6 / cells + 60))
        return {**_RUN, "mesh": "quad" if cells < 60_000 and rng.random() < 0.3 else "voronoi", "cells": cells,
                "water": water, "radius": round(_log(rng, 0.04, 0.3), 3), "cfl": rng.choice([0.8, 0.8, 0.9, 0.5]),
                "seconds": round({"lake": 0.13, "dam": 0.06, "wet": 0.025}[water] * steps, 3), "windows": rng.randint(1, 4),
                "compensated": rng.random() < 0.8, "clamp": rng.random() < 0.2}
    if kind == "phases":
        return {"kind": kind, "cells": int(_log(rng, 5000, 200_000)), "phases": rng.randint(2, 4),
                "seconds": round(_log(rng, 1.0, 20.0), 3), "inflows": rng.randint(1, 20)}
    if kind == "channel":
        return {"kind": kind, "cells": rng.randint(80, 900), "across": rng.randint(5, 60),
                "seconds": round(_log(rng, 20.0, 600.0), 2), "windows": rng.randint(1, 4)}
    if kind == "batch":
        members = rng.choice([1, 2, 5, 11, 16, 24])
        rain = members == 1 or rng.random() < 0.4
        return {"kind": kind, "members": members, "cells": int(_log(rng, 4000, 900_000) / members ** 0.8),
                "spread": round(rng.uniform(1.0, 4.0), 2), "rain": rain, "seconds": round(_log(rng, 3.0, 30.0), 3)}
    cells = int(_log(rng, 5000, 250_000))
    return {"kind": kind, "cells": cells, "steps": rng.randint(10, 100), "every": rng.choice([8, 25, 40, 50]),
            "gauges": rng.randint(5, 200), "knots": rng.randint(3, 32)}


# -- meshes -----------------------------------------------------------------------------------
def _reflected(patch_cells: int, per_side: int, side: float, seed: int):
    """The patch of ``patch_cells`` Voronoi cells over [0, side]^2, continued by reflection to per_side^2 patches."""
    mesh = voronoi_mesh(patch_cells, side, seed)
    verts = np.where(np.abs(mesh.verts - side) < 1e-7 * side, side, np.where(mesh.verts < 1e-7 * side, 0.0, mesh.verts))
    degree = np.diff(mesh.offsets)
    # a vertex on a seam is the same vertex in both patches: on x = 0 or x = side its column decides
    on = [(verts[:, a] == 0.0, verts[:, a] == side) for a in (0, 1)]
    coords, keys, faces, sizes = [], [], [], []
    n_v = verts.shape[0]
    reverse = np.concatenate([np.arange(e - 1, s - 1, -1) for s, e in zip(mesh.offsets[:-1], mesh.offsets[1:])])
    for i in range(per_side):
        for j in range(per_side):
            x = side * i + (verts[:, 0] if i % 2 == 0 else side - verts[:, 0])
            y = side * j + (verts[:, 1] if j % 2 == 0 else side - verts[:, 1])
            coords.append(np.column_stack([x, y]))
            # the seam vertex belongs to the patch before the seam
            left = on[0][0] if i % 2 == 0 else on[0][1]
            down = on[1][0] if j % 2 == 0 else on[1][1]
            pi, pj = np.where(left & (i > 0), i - 1, i), np.where(down & (j > 0), j - 1, j)
            key = (pi * per_side + pj).astype(np.int64) * n_v + np.arange(n_v)
            keys.append(key)
            order = reverse if (i + j) % 2 else slice(None)  # a reflection turns the ring around
            faces.append(key[mesh.faces[order]])
            sizes.append(degree)
    key, coord = np.concatenate(keys), np.concatenate(coords)
    ids, first, flat = np.unique(np.concatenate([key, *faces]), return_index=True, return_inverse=True)
    offsets = np.zeros(per_side * per_side * degree.size + 1, np.int32)
    np.cumsum(np.concatenate(sizes), out=offsets[1:])
    return coord[first], flat[key.size :].astype(np.int32), offsets


@functools.lru_cache(maxsize=None)
def _geometry(kind: str, cells: int, across: int = 0):
    """Hilbert-ordered geometry on a flat bed, and the length of its longer side."""
    if kind == "voronoi":
        per_side = max(1, math.ceil(math.sqrt(cells / PATCH_CELLS)))
        patch = round(cells / per_side**2)
        verts, faces, offsets = _reflected(patch, per_side, SPACING * math.sqrt(patch), seed=17 + cells % 97)
        geom = build_geometry(verts, faces, offsets, zb_from_file=np.zeros(offsets.size - 1, np.float32))
        side = SPACING * math.sqrt(patch) * per_side
    elif kind == "quad":
        nx = max(8, 2 * round(math.sqrt(cells / 2)))
        m = quad_grid(nx, max(4, round(cells / nx)), 2.0)
        geom = build_geometry(m.verts.astype(np.float32), m.faces.reshape(-1, 4), zb_from_file=np.zeros(m.n_cells, np.float32))
        side = 2.0 * nx
    else:
        m = channel_grid(cells, across, 10.0 * cells, 10.0 * across)
        geom = build_geometry(m.verts, m.faces, m.offsets, zb_from_file=np.zeros(m.n_cells, np.float32))
        side = 10.0 * cells
    return hilbert_reorder(geom, verbose=False)[0], side


def _f32(a) -> np.ndarray:
    return np.ascontiguousarray(a, np.float32)


# -- inputs from the seed: one dict of host arrays per mesh ---------------------------------------
def _scene(case: dict, seed: int, member: int = 0) -> dict:
    rng = np.random.default_rng([seed, member])
    kind = case["kind"]
    cells = case["cells"]
    if kind == "batch" and case["members"] > 1:  # sizes spread evenly over their logarithm
        f = (member + 0.5) / case["members"] - 0.5
        cells = int(cells * case["spread"] ** (2 * f))
    if kind == "channel":
        geom, side = _geometry("channel", cells, case["across"])
    else:
        geom, side = _geometry(case.get("mesh", "voronoi"), cells)
    xy = geom.world_centroid
    bed_seed = int(rng.integers(1 << 30))
    n = rng.uniform(0.025, 0.045, geom.N)
    hu = hv = np.zeros(geom.N)
    s: dict = {"area": geom.area.astype(np.float64)}
    if kind == "channel":
        slope = rng.uniform(0.8e-3, 1.2e-3)
        zb = 10.0 - slope * xy[:, 0]
        across = math.pi * xy[:, 1] / (10.0 * case["across"])
        h = rng.uniform(0.3, 0.6) + rng.uniform(0.02, 0.05) * np.cos(across)  # a little higher at one bank
        n = np.full(geom.N, rng.uniform(0.028, 0.032))
        width = 10.0 * case["across"]
        s["open"] = [select_boundary_edges(geom, [(x, 0.0), (x, width)], 2.5) for x in (0.0, side)]
        s["inflow"] = rng.uniform(0.3, 0.9)  # m^2/s per unit width
        s["normal"] = math.sqrt(slope) / float(n[0])
    elif case.get("water") == "lake":
        zb = gaussian_bumps(xy, side, count=6, seed=bed_seed)
        tilt = rng.uniform(0.02, 0.06) * np.cos(math.pi * xy[:, 0] / side)
        h = np.maximum(1.0 + tilt - zb, 0.0)
    else:
        zb = fractal_dem(xy, side, relief=20.0 if side > 1000.0 else 1.0, beta=2.0, seed=bed_seed)
        if case.get("water") == "wet":
            wave = rng.uniform(0.2, 0.4) * np.sin(2 * math.pi * (xy[:, 0] + 0.5 * xy[:, 1]) / side + rng.uniform(0, 6))
            h = 1.0 + wave + 0.1 * rng.random(geom.N)
        elif kind == "batch" and case["rain"]:
            h = rng.uniform(0.002, 0.02, geom.N)
        else:
            centre = side * rng.uniform(0.42, 0.58, 2)
            r = np.hypot(xy[:, 0] - centre[0], xy[:, 1] - centre[1])
            radius = {"run": case.get("radius"), "phases": 0.05, "batch": 0.06, "gradient": 0.1}[kind]
            depth = {"run": 4.0, "phases": 1.0, "batch": 1.0, "gradient": 1.0}[kind]
            h = np.where(r <= radius * side, depth * rng.uniform(0.9, 1.1), 0.0)
            s["near"] = np.argsort(r)
    s.update(geom=with_bed(geom, _f32(zb)), h=_f32(h), hu=_f32(hu), hv=_f32(hv), n=_f32(n))
    if kind == "phases":
        rates = np.zeros((case["phases"], geom.N))
        at = rng.choice(s["near"][: geom.N // 20], case["inflows"], replace=False)
        rates[:, at] = rng.uniform(2.0, 30.0, (case["phases"], at.size))
        s["rates"] = [_f32(r) for r in rates]
    if kind == "batch":
        s["rain"] = _f32(0.05 / 3600.0 * s["area"]) if case["rain"] else None
        cell = int(np.argmax(zb)) if case["rain"] else int(s["near"][0])
        s["hydro"] = (cell, _f32([0.0, 0.6, 1.1, 1.9]) * np.float32(case["seconds"]), _f32(rng.uniform(10.0, 200.0, 4)))
    if kind == "gradient":
        s["gauges"] = np.sort(rng.choice(s["near"][: max(case["gauges"], geom.N // 8)], case["gauges"], replace=False))
        s["n_true"] = _f32(rng.uniform(0.02, 0.06, geom.N))
        s["n"] = np.full(geom.N, 0.035, np.float32)
        t = np.linspace(0.0, 1.2 * 0.03 * case["steps"], case["knots"])
        s["hydro"] = (int(s["near"][0]), _f32(t), _f32(rng.uniform(20.0, 60.0, case["knots"])))
    return s


def _hydrograph(s: dict) -> Hydrograph:
    cell, t, q = s["hydro"]
    return Hydrograph(cells=np.array([cell]), knot_t=t, knot_q=q)


# -- the passes -----------------------------------------------------------------------------------
def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "batch":
        scenes = [_scene(case, seed, i) for i in range(case["members"])]
        members = [BatchMember(s["geom"], s["h"], s["hu"], s["hv"], s["n"], source_rate=s["rain"],
                               hydrographs=[_hydrograph(s)]) for s in scenes]
        return {"case": case, "solver": BatchedSolver(members, cfl=0.8)}
    s = _scene(case, seed)
    if kind == "gradient":
        problem = GaugeCalibration(s["geom"], s["h"], s["hu"], s["hv"], gauges=s["gauges"], steps=case["steps"],
                                   hydrographs=[_hydrograph(s)], checkpoint_every=case["every"], dt_max=1.0, dt_init=0.05)
        problem.cut_depth = FILM_DEPTHS * DRY_TOL
        z, q = s["geom"].zb.astype(np.float32), s["hydro"][2]
        problem.observe(s["n_true"], z, q)
        return {"case": case, "problem": problem, "n": s["n"], "z": z, "q": q}
    opened = {"open_edges": s["open"]} if kind == "channel" else {}
    solver = SWESolverB200Resident(s["geom"], None, s["h"], s["hu"], s["hv"], s["n"], cfl=case.get("cfl", 0.8), **opened)
    if kind == "channel":
        up, down = (e.size for e in s["open"])
        solver.set_open_conditions(np.repeat([OPEN_INFLOW, OPEN_NORMAL], [up, down]).astype(np.uint32),
                                   np.repeat([s["inflow"], s["normal"]], [up, down]).astype(np.float32))
    if kind == "run":
        solver.compensated, solver.track_clamp = case["compensated"], case["clamp"]
    return {"case": case, "solver": solver, "rates": s.get("rates")}


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "gradient":
        problem = state["problem"]
        loss = problem.loss(state["n"], state["z"], state["q"])
        gn, gz, gq = problem.gradient()
        return {"loss": loss, "n": gn, "z": gz, "q": gq}
    solver = state["solver"]
    if kind == "batch":
        solver.run(case["seconds"], 1.0, 0.01, case["seconds"] / 2)
        every = range(case["members"])
        return {"h": np.concatenate([solver.download_h(i) for i in every]),
                "hu": np.concatenate([solver.download_hu(i) for i in every]),
                "hv": np.concatenate([solver.download_hv(i) for i in every])}
    settings = {"dt_max": case.get("dt_max", 1.0), "dt_init": min(0.01, case.get("dt_max", 1.0)), "cfl_interval": 10,
                "progress": False}
    if kind == "phases":
        length = case["seconds"]
        for k, rate in enumerate(state["rates"]):
            snaps, _ = solver.run(t_end=(k + 1) * length, output_interval_s=length, source_rate=rate, resume=k > 0,
                                  t_start=k * length, **settings)
    else:
        snaps, _ = solver.run(t_end=case["seconds"], output_interval_s=case["seconds"] / case["windows"], **settings)
    out = {"h": snaps[-1], "hu": solver.download_hu(), "hv": solver.download_hv()}
    if kind == "channel":
        out["volume"] = solver.download_open_volumes()
    return out


def work(case: dict) -> dict:
    """One read of the mesh and the state and one write of the state per step, over the cells that water can reach."""
    kind = case["kind"]
    n, seconds, wet = case["cells"], case.get("seconds", 0.0), 1.0
    if kind == "run":  # steps a second of each kind of water, from its CFL bound
        if case["water"] == "dam":
            wet = min(1.0, 4.0 * case["radius"] ** 2 + 0.01)
        steps = seconds * max({"lake": 7.5, "dam": 18.0, "wet": 44.0}[case["water"]], 1.0 / case["dt_max"])
    elif kind == "phases":
        steps, wet = case["phases"] * seconds * 13.0, 0.02
    elif kind == "channel":
        n, steps = n * case["across"], seconds * 1.3
    elif kind == "batch":
        n, wet = n * case["members"], 1.0 if case["rain"] else 0.02
        steps = seconds * (3.0 if case["rain"] else 9.0)
    else:
        steps, wet = 3 * case["steps"], 0.05  # forward, forward again, reverse
    # per cell: 3 edges of 28 B, 6 slots of 4 B, area, roughness and pointer, four words in and out
    return {"bytes": steps * wet * n * (84 + 24 + 12 + 32) + 12 * n, "flops": steps * wet * n * 1400}


# -- the same passes in float64 ---------------------------------------------------------------------
def _device() -> str:
    return "cuda" if torch.cuda.is_available() else "cpu"


def _sqrt(x):  # derivative 0 at 0
    pos = x > 0
    return torch.where(pos, torch.sqrt(torch.where(pos, x, torch.ones_like(x))), torch.zeros_like(x))


def _quotient(num, den, ok):
    return torch.where(ok, num / torch.where(ok, den, torch.ones_like(den)), torch.zeros_like(num))


class _Exact:
    """The Heun step of one mesh in float64 torch, over all cells and edges."""

    def __init__(self, s: dict, cfl: float = 0.8, cut: float = 0.0) -> None:
        g = s["geom"]
        self.t = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=_device())
        self.i = lambda a: torch.as_tensor(np.asarray(a, np.int64), device=_device())
        self.cl, cr = self.i(g.edge_cellL), np.asarray(g.edge_cellR, np.int64)
        self.wall, self.cr = self.i(cr < 0).bool(), self.i(np.maximum(cr, 0))
        self.inner = torch.nonzero(~self.wall).flatten()
        self.nx, self.ny, self.len = self.t(g.edge_nx), self.t(g.edge_ny), self.t(g.edge_len)
        self.dzl, self.dzr = self.t(g.edge_dzL), self.t(g.edge_dzR)
        self.area, self.n = self.t(g.area), self.t(s["n"])
        self.state = tuple(self.t(s[k]) for k in ("h", "hu", "hv"))
        self.cfl, self.cut = cfl, cut
        self.sources = None  # (cells, function of the clock: depth rate)
        self.opened = None
        if "open" in s:
            up, down = (self.i(e) for e in s["open"])
            self.opened = (up, down, float(np.float32(s["inflow"])), float(np.float32(s["normal"])))
            self.volume = torch.zeros(2, 2, dtype=torch.float64, device=_device())

    def hold(self, h, *vals):  # no derivative through thin depths
        return tuple(torch.where(h < self.cut, v.detach(), v) for v in vals) if self.cut > 0.0 else vals

    def velocity(self, h, q):
        h2 = h * h
        return torch.where(h > DRY_TOL, 2.0 * h * q / (h2 + torch.clamp(h2, min=(FILM_DEPTHS * DRY_TOL) ** 2)), 0.0 * h)

    def ghosts(self, hL, huL, hvL, hR, huR, hvR):
        up, down, q, k = self.opened
        for e in (up, down):
            nx, ny, h = self.nx[e], self.ny[e], hL[e]
            u, v = self.velocity(h, huL[e]), self.velocity(h, hvL[e])
            un, ut = u * nx + v * ny, v * nx - u * ny
            if e is up:
                riemann, root = un + 2.0 * torch.sqrt(GRAVITY * h), math.sqrt(GRAVITY)
                x = torch.maximum(torch.full_like(h, (q / (2.0 * root)) ** (1.0 / 3.0)), riemann / (2.0 * root))
                for _ in range(4):
                    f = 2.0 * root * x - q / (x * x) - riemann
                    x = torch.maximum(x - f / (2.0 * root + 2.0 * q / x**3), 0.5 * x)
                h = x * x
                un, ut = -q / h, 0.0 * h
            else:
                un = k * h ** (2.0 / 3.0)
            hR, huR, hvR = (a.index_copy(0, e, b) for a, b in ((hR, h), (huR, h * (un * nx - ut * ny)), (hvR, h * (un * ny + ut * nx))))
        return hR, huR, hvR

    def fluxes(self, h, hu, hv):
        nx, ny, wall = self.nx, self.ny, self.wall
        hL, huL, hvL = self.hold(h[self.cl], h[self.cl], hu[self.cl], hv[self.cl])
        dot = huL * nx + hvL * ny
        hR = torch.where(wall, hL, h[self.cr])
        huR = torch.where(wall, huL - 2.0 * dot * nx, hu[self.cr])
        hvR = torch.where(wall, hvL - 2.0 * dot * ny, hv[self.cr])
        if self.opened:
            hR, huR, hvR = self.ghosts(hL, huL, hvL, hR, huR, hvR)
        hR, huR, hvR = self.hold(hR, hR, huR, hvR)
        side = []
        for a, b, c, dz in ((hL, huL, hvL, self.dzl), (hR, huR, hvR, self.dzr)):
            hs = torch.clamp(a - dz, min=0.0)
            (hs,) = self.hold(hs, hs)
            qx, qy = hs * self.velocity(a, b), hs * self.velocity(a, c)
            un, ut = self.velocity(hs, qx * nx + qy * ny), self.velocity(hs, qy * nx - qx * ny)
            side.append((hs, un, ut, _sqrt(hs), torch.clamp(hs / DRY_TOL - 1.0, 0.0, 1.0)))
        (hl, unl, utl, rl, wl), (hr, unr, utr, rr, wr) = side
        root = math.sqrt(GRAVITY)
        cl, cr = root * rl, root * rr
        mean = _quotient(rl * unl + rr * unr, rl + rr, rl + rr > 1e-12)
        cm = _sqrt(GRAVITY * 0.5 * (hl + hr))
        dl, dr = (1.0 - wl) * wr, (1.0 - wr) * wl
        SL = (1.0 - dl - dr) * torch.minimum(unl - cl, mean - cm) + dl * (unr - 2.0 * cr) + dr * (unl - cl)
        SR = (1.0 - dl - dr) * torch.maximum(unr + cr, mean + cm) + dl * (unr + cr) + dr * (unl + 2.0 * cl)
        den = hr * (unr - SR) - hl * (unl - SL)
        SM = _quotient(SL * hr * (unr - SR) - SR * hl * (unl - SL), den, den.abs() > 1e-12)
        left = (SL >= 0) | (SM >= 0)
        star = ~(SL >= 0) & (left | (SR >= 0))
        hx, un, ut, S = (torch.where(left, a, b) for a, b in ((hl, hr), (unl, unr), (utl, utr), (SL, SR)))
        d = S - SM
        k = hx * (S - un) / torch.where(d.abs() > 1e-14, d, torch.full_like(d, 1e-14))
        Fh = hx * un + torch.where(star, S * (k - hx), 0.0 * hx)
        Fn = hx * un * un + 0.5 * GRAVITY * hx * hx + torch.where(star, S * (k * SM - hx * un), 0.0 * hx)
        Ft = hx * un * ut + torch.where(star, S * (k - hx) * ut, 0.0 * hx)
        Fm = torch.where(wall, 0.0 * Fh, Fh)
        if self.opened:
            up, down, q, _ = self.opened
            Fm = Fm.index_fill(0, up, -q).index_copy(0, down, torch.clamp(Fh[down], min=0.0))
        Fx, Fy = Fn * nx - Ft * ny, Fn * ny + Ft * nx
        bl, br = 0.5 * GRAVITY * (hL * hL - hl * hl), 0.5 * GRAVITY * (hR * hR - hr * hr)
        live = ~((hL < DRY_TOL) & (hR < DRY_TOL))
        if self.opened:
            live = live.index_fill(0, self.opened[0], True)
        w = self.len * live
        speed = torch.maximum(SL.abs(), SR.abs()) * w
        return Fm * w, (Fx + bl * nx) * w, (Fy + bl * ny) * w, (Fx + br * nx) * w, (Fy + br * ny) * w, speed

    def gather(self, to_left, to_right):
        inner = self.inner
        return torch.zeros_like(self.area).index_add(0, self.cl, to_left).index_add(0, self.cr[inner], to_right[inner])

    def bound(self, speed) -> float:
        lam = self.gather(speed.detach(), speed.detach())
        ok = (lam > 1e-30) & (self.area > 1e-10)
        return float((self.cfl * self.area[ok] / lam[ok]).min()) if bool(ok.any()) else 1e30

    def stage(self, h, hu, hv, dt):
        w0, w1, w2, w3, w4, speed = self.fluxes(h, hu, hv)
        if self.opened:
            for k, e in enumerate(self.opened[:2]):
                v = 0.5 * dt * w0[e]
                self.volume[k] += torch.stack([torch.clamp(v, min=0.0).sum(), torch.clamp(-v, min=0.0).sum()])
        dti = dt / self.area
        sh, su, sv = self.gather(w0, -w0), self.gather(w1, -w3), self.gather(w2, -w4)
        h, hu, hv = self.hold(h, h, hu, hv)
        h = torch.clamp(h - dti * sh, min=0.0)
        wet = h >= DRY_TOL
        e = FILM_DEPTHS * DRY_TOL
        x = torch.where(wet, h, torch.ones_like(h))
        drag = torch.where(x < e, 1.0 / (1.0 + dt * (e * e - x * x) / (2.0 * x * x) * math.sqrt(GRAVITY / e)), torch.ones_like(x))
        drag, x = self.hold(x, drag, x)
        hu, hv = (hu - dti * su) * drag, (hv - dti * sv) * drag
        speed_of = _sqrt((hu / x) ** 2 + (hv / x) ** 2)
        den = 1.0 + dt * GRAVITY * self.n * self.n * speed_of / x ** (4.0 / 3.0)
        return h, torch.where(wet, hu / den, 0.0 * hu), torch.where(wet, hv / den, 0.0 * hv), speed

    def step(self, h, hu, hv, dt, clock):
        a = self.stage(h, hu, hv, dt)
        b = self.stage(*a[:3], dt)
        h = 0.5 * (h + b[0])
        wet = h >= DRY_TOL
        hu, hv = (torch.where(wet, 0.5 * (x + y), 0.0 * h) for x, y in ((hu, b[1]), (hv, b[2])))
        if self.sources:
            cells, rate = self.sources
            h = h.index_add(0, cells, dt * rate(clock))
        return h, hu, hv, b[3]

    def source_bound(self, h, hu, hv) -> float:
        """The bound of the cells a source has filled, from their depth and their neighbours'."""
        cells = self.sources[0]
        wet = h >= DRY_TOL
        other_dry = ~wet[self.cr] & ~self.wall
        hs = torch.where(wet, h, torch.ones_like(h))
        u, c = torch.hypot(hu, hv) / hs, torch.sqrt(GRAVITY * hs)
        lam = self.gather((u[self.cl] + torch.where(other_dry, 2.0, 1.0) * c[self.cl]) * self.len,
                          (u[self.cr] + torch.where(~wet[self.cl], 2.0, 1.0) * c[self.cr]) * self.len)
        b = (self.cfl * self.area / lam)[cells][wet[cells]]
        return float(b.min()) if b.numel() else 1e30

    @staticmethod
    def ticks(bound: float, dt_max: int, dry: int, left: int) -> int:
        t = dry if bound >= 1e10 else int(min(bound, dt_max / TICKS) * TICKS)
        return min(t, dt_max, left)

    @torch.no_grad()
    def advance(self, start: float, stops: list[float], dt_max: float, dt_init: float) -> None:
        now, top, dry = round(start * TICKS), int(dt_max * TICKS), int(min(dt_init, dt_max) * TICKS)
        bound = self.bound(self.fluxes(*self.state)[5])
        for stop in stops:
            end = round(stop * TICKS)
            while now < end:
                t = self.ticks(bound, top, dry, end - now)
                if t <= 0:
                    raise RuntimeError("the clock stalled")
                *state, speed = self.step(*self.state, t / TICKS, now / TICKS)
                self.state, bound = tuple(state), self.bound(speed)
                if self.sources:
                    bound = min(bound, self.source_bound(*self.state))
                now += t

    def misfit(self, s: dict, steps: int, observed, q):
        """The gauge misfit of ``steps`` steps (or, without observations, the gauge depths)."""
        gauges = self.i(s["gauges"])
        cell, kt, _ = s["hydro"]
        scale = float(np.float32(1.0 / s["geom"].area[cell]))
        self.sources = (self.i([cell]), lambda t: (scale * _interpolate(kt, q, t)).reshape(1))
        now, state, total, seen = 0, self.state, 0.0, []
        with torch.no_grad():
            bound = self.bound(self.fluxes(*state)[5])
        for k in range(steps):
            t = self.ticks(bound, TICKS, int(0.05 * TICKS), 1 << 62)
            *state, speed = self.step(*state, t / TICKS, now / TICKS)
            with torch.no_grad():
                bound = min(self.bound(speed), self.source_bound(*state))
            now += t
            depth = state[0][gauges]
            seen.append(depth.detach())
            if observed is not None:
                total = total + ((depth - observed[k]) ** 2).sum()
        return seen if observed is None else total


def _interpolate(kt, q, t: float):
    if not t > kt[0]:
        return q[0]
    if not t < kt[-1]:
        return q[-1]
    i = min(int(np.searchsorted(kt, t, side="right")) - 1, len(kt) - 2)
    return q[i] + (q[i + 1] - q[i]) * ((t - float(kt[i])) / (float(kt[i + 1]) - float(kt[i])))


def _windows(case: dict) -> list[float]:
    every = round(case["seconds"] / case["windows"] * TICKS)
    end = round(case["seconds"] * TICKS)
    return [k * every / TICKS for k in range(1, case["windows"] + 1) if k * every < end] + [end / TICKS]


def exact(case: dict, seed: int):
    kind = case["kind"]
    numpy = lambda *ts: [t.detach().cpu().numpy() for t in ts]  # noqa: E731
    if kind == "batch":
        if case["members"] > 6:
            return None  # one mesh after the other takes too long
        parts = []
        for i in range(case["members"]):
            s = _scene(case, seed, i)
            m = _Exact(s)
            (cell, kt, kq), inv = s["hydro"], (1.0 / s["geom"].area).astype(np.float32)
            rate = np.zeros(m.area.numel(), np.float32) if s["rain"] is None else s["rain"] * inv
            live = np.flatnonzero((rate != 0) | (np.arange(rate.size) == cell))
            steady, share = m.t(rate[live]), m.t(np.where(live == cell, inv[live], 0.0))
            m.sources = (m.i(live), lambda t, a=steady, b=share, k=kt, q=kq: a + b * float(_interpolate(k, q, t)))
            m.advance(0.0, [round(case["seconds"] / 2 * TICKS) / TICKS, round(case["seconds"] * TICKS) / TICKS], 1.0, 0.01)
            parts.append(numpy(*m.state))
        return {k: np.concatenate([p[j] for p in parts]) for j, k in enumerate(("h", "hu", "hv"))}
    s = _scene(case, seed)
    if kind == "gradient":
        if case["cells"] * case["steps"] > 4_000_000:
            return None  # the tape of every operation is too large
        z, q = s["geom"].zb.astype(np.float32), s["hydro"][2]
        with torch.no_grad():
            truth = _Exact({**s, "n": s["n_true"]})
            seen = truth.misfit(s, case["steps"], None, truth.t(q))
        m = _Exact(s, cut=FILM_DEPTHS * DRY_TOL)
        m.n.requires_grad_(True)
        bed, knots = m.t(z).requires_grad_(True), m.t(q).requires_grad_(True)
        zl = bed[m.cl]
        zr = torch.where(m.wall, zl, bed[m.cr])
        face = torch.maximum(zl, zr)
        m.dzl, m.dzr = face - zl, torch.where(m.wall, 0.0 * zl, face - zr)
        loss = m.misfit(s, case["steps"], seen, knots)
        loss.backward()
        return {"loss": float(loss.detach()), **dict(zip(("n", "z", "q"), numpy(m.n.grad, bed.grad, knots.grad)))}
    m = _Exact(s, cfl=case.get("cfl", 0.8))
    if kind == "phases":
        inv = (1.0 / s["geom"].area).astype(np.float32)
        for k, rate in enumerate(s["rates"]):
            live = np.flatnonzero(rate)
            steady = m.t(rate[live] * inv[live])
            m.sources = (m.i(live), lambda t, a=steady: a)
            m.advance(k * case["seconds"], [(k + 1) * case["seconds"]], 1.0, 0.01)
    else:
        dt_max = case.get("dt_max", 1.0)
        m.advance(0.0, _windows(case), dt_max, 0.01)
    out = dict(zip(("h", "hu", "hv"), numpy(*m.state)))
    if kind == "channel":
        out["volume"] = m.volume.cpu().numpy()
    return out
