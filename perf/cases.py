"""What a user of this framework has it do, as measurable cases.

Every case goes through the public Python binding or the C ABI (vare_gb300.flip). The kinds:

  step        particles in host memory -> one FLIPMethod::advanceOneStep -> particles in host
              memory, as a host application that owns its particles calls it each frame (the
              end-to-end measurement of bench.py)
  batch       the same for several independent simulations stepped together (the serving layer's
              round)
  grid        SparseFrame::buildFromPoints and P2G over resident particles, and the grid read back
  project     the pressure projection of a P2G grid: system, solve, velocity update
  splat       the surface and velocity splat that starts a frame's post-processing
  redistance  the redistancing of a surface field given by the caller
  vdb         a frame's surface and velocity as VDB leaf blocks
  scan        the device prefix sum on its own

Scenes are the repository's: a dam break (block and falling sphere) in a cubic or ragged box,
and a sparse wide tank with a wave column and a static box obstacle, 8 jittered particles per
cell, solid walls. Sizes go from the tests' small scenes (24^3) to the 256^3 benchmark scene.
Particles move with a smooth swirl (tangential at the walls) so that every step has a pressure
to solve for; positions, speeds and phases come from the seed.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from vare_gb300 import flip

PPC = 8
SURF_BACKGROUND = 10.0  # the surface field outside the active tiles (FLIPMethod.cu:30)
EXACT_CELLS = 60_000_000  # dense cells up to which exact() solves a projection


def listed():
    return [
        # a test or preview scene: a step is all launches and waits
        step("step_dam24_plain", 24, 24, 24, "plain", fx=0.4, fy=0.55, sphere=0.15),
        # the 64^3 dam break, the repository's first configuration
        step("step_dam64_plain", 64, 64, 64, "plain", fx=0.4, fy=0.6),
        # a request of the serving mix on its own, ragged box, midpoint advection
        step("step_dam96_mixed_rk2", 110, 90, 97, "mixed", fx=0.45, fy=0.5, sphere=0.13, rk2=True),
        # the benchmark's scene in both solver forms: 24.6 M particles
        step("step_dam256_plain", 256, 256, 256, "plain", fx=0.35, fy=0.5, sphere=0.12),
        step("step_dam256_mixed", 256, 256, 256, "mixed", fx=0.35, fy=0.5, sphere=0.12),
        # the large sparse domain at 5/8 of its edge: 39 M particles, about 5 % of the tiles, a collider
        {"name": "step_tank640_mixed", "kind": "step", "scene": "tank", "nx": 640, "ny": 320, "nz": 640,
         "solver": "mixed", "depth": 8, "rk2": False},
        # a round of the serving layer: requests of 32 .. 96 cells per edge
        {"name": "batch_mixed", "kind": "batch", "scene": "dam", "count": 8, "lo": 32, "hi": 96, "fx": 0.5, "fy": 0.5,
         "sphere": 0.0, "solver": "mixed", "rk2": False},
        # particles to grid at a ragged size, the grid fields read back (motion blur, whitewater)
        {"name": "grid_dam150", "kind": "grid", "scene": "dam", "nx": 150, "ny": 121, "nz": 170, "fx": 0.5, "fy": 0.5,
         "sphere": 0.1},
        # the projection alone at a production size
        {"name": "project_dam192_mixed", "kind": "project", "scene": "dam", "nx": 192, "ny": 192, "nz": 192, "fx": 0.4,
         "fy": 0.5, "sphere": 0.12, "solver": "mixed"},
        # the two stages that make up most of a frame's post-processing
        {"name": "splat_dam128", "kind": "splat", "scene": "dam", "nx": 128, "ny": 128, "nz": 128, "fx": 0.4, "fy": 0.5,
         "sphere": 0.12},
        {"name": "redistance_dam256", "kind": "redistance", "scene": "dam", "nx": 256, "ny": 256, "nz": 256, "fx": 0.35,
         "fy": 0.5, "sphere": 0.12},
        # a frame's fields on their way to OpenVDB
        {"name": "vdb_dam128", "kind": "vdb", "scene": "dam", "nx": 128, "ny": 128, "nz": 128, "fx": 0.4, "fy": 0.5,
         "sphere": 0.12},
    ]


def step(name, nx, ny, nz, solver, fx, fy, sphere=0.0, rk2=False):
    return {"name": name, "kind": "step", "scene": "dam", "nx": nx, "ny": ny, "nz": nz, "solver": solver, "fx": fx,
            "fy": fy, "sphere": sphere, "rk2": rk2}


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "step", "step", "batch", "grid", "project", "project", "splat", "redistance", "vdb",
                       "scan"])
    if kind == "scan":
        return {"kind": "scan", "n": log(1000, 100_000_000)}
    solver = rng.choice(["plain", "mixed"])
    if kind == "step" and rng.random() < 0.25:
        n = log(128, 512)
        return {"kind": kind, "scene": "tank", "nx": n, "ny": max(48, n // 2 + rng.randint(-8, 8)), "nz": n + rng.randint(-9, 9),
                "solver": solver, "depth": rng.randint(5, 12), "rk2": False}
    c = {"kind": kind, "scene": "dam", "fx": round(rng.uniform(0.3, 0.5), 3), "fy": round(rng.uniform(0.3, 0.5), 3),
         "sphere": round(rng.choice([0.0, rng.uniform(0.08, 0.13)]), 3)}
    if kind == "batch":
        lo = log(28, 64)
        return dict(c, count=rng.randint(2, 10), lo=lo, hi=lo + rng.randint(4, 40), solver="mixed", rk2=False)
    hi = 128 if kind in ("splat", "vdb") else 230
    n = log(24, hi)
    for k in ("nx", "ny", "nz"):
        c[k] = max(20, int(n * rng.uniform(0.8, 1.08)))
    if kind in ("step", "project"):
        c["solver"] = solver
    if kind == "step":
        c["rk2"] = rng.random() < 0.25
    return c


# ---- scenes ------------------------------------------------------------------------------

def frame(case):
    """The simulation grid: the requested cells padded to a multiple of 4 per axis."""
    return tuple((case[k] + 3) // 4 * 4 for k in ("nx", "ny", "nz"))


def members(case):
    """The simulations of a case: itself, or the batch's (edges spread over lo .. hi)."""
    if case["kind"] != "batch":
        return [case]
    out = []
    for k in range(case["count"]):
        e = int(round(case["lo"] * (case["hi"] / case["lo"]) ** (k / max(1, case["count"] - 1))))
        out.append(dict(case, kind="step", nx=e, ny=e - k % 3, nz=e + k % 2))
    return out


def tank_box(case):
    """The tank's static obstacle: lo and hi corners in voxels."""
    nx, ny, nz = frame(case)
    # no cell centre lies on a face
    return ((round(0.45 * nx) + 0.25, -2.0, round(0.3 * nz) + 0.25),
            (round(0.55 * nx) - 0.25, round(0.06 * ny) + 0.25, round(0.7 * nz) - 0.25))


def filled(case):
    """(nz, ny, nx) mask of the cells that hold particles, as (mask, j extent)."""
    nx, ny, nz = frame(case)
    X = ((torch.arange(nx, device="cuda") + 0.5) / nx).view(1, 1, nx)
    Z = ((torch.arange(nz, device="cuda") + 0.5) / nz).view(nz, 1, 1)
    if case["scene"] == "tank":
        top = max(case["depth"], int(0.3 * ny))
        j = torch.arange(top, device="cuda").view(1, top, 1)
        m = (j < case["depth"]) | ((X < 0.04) & (j < int(0.3 * ny)))
        lo, hi = tank_box(case)
        i = torch.arange(nx, device="cuda").view(1, 1, nx) + 0.5
        k = torch.arange(nz, device="cuda").view(nz, 1, 1) + 0.5
        away = 3.5  # no particle reaches the obstacle within the step
        near = (i > lo[0] - away) & (i < hi[0] + away) & (k > lo[2] - away) & (k < hi[2] + away) & (j + 0.5 < hi[1] + away)
        return (m & ~near).expand(nz, top, nx), top
    Y = ((torch.arange(ny, device="cuda") + 0.5) / ny).view(1, ny, 1)
    m = (X < case["fx"]) & (Y < case["fy"]) & (Z < 2)
    if case["sphere"]:
        m = m | ((X - 0.7) ** 2 + (Y - 0.8) ** 2 + (Z - 0.5) ** 2 < case["sphere"] ** 2)
    return m, ny


def time_step(case):
    return 1.0 / 240.0 * 64.0 / max(frame(case))


def particles(case, seed):
    """Positions and velocities on the GPU, (N, 3) float32 in voxels and voxels per second."""
    nx, ny, nz = frame(case)
    gen = torch.Generator("cuda").manual_seed(seed)
    mask, _ = filled(case)
    kji = mask.nonzero()
    ijk = kji.flip(1).to(torch.float32)
    n = ijk.shape[0]
    pos = torch.rand(n, PPC, 3, generator=gen, device="cuda")
    pos *= 0.999  # no position rounds up into the next cell
    pos += ijk.view(n, 1, 3)
    pos = pos.view(-1, 3)
    par = torch.rand(6, generator=gen, device="cuda").tolist()
    amp = (0.4 + 0.4 * par[0]) / time_step(case)
    vel = torch.empty_like(pos)
    X, Y, Z = (pos[:, a] * (math.pi / f) for a, f in enumerate((nx, ny, nz)))
    vel[:, 0] = amp * torch.sin(X) * torch.cos(Y + 0.3 * par[1])
    vel[:, 1] = -amp * torch.cos(X + par[2]) * torch.sin(Y)
    vel[:, 2] = 0.5 * amp * torch.sin(Z) * torch.cos(2 * X + 3 * par[3]) * (0.5 + par[4])
    vel *= 1.0 + 0.1 * (torch.rand(vel.shape, generator=gen, device="cuda") - 0.5)
    return pos, vel


def make_sim(case):
    n = max(frame(case))
    params = dict(ext_force=(0.0, -9.8, 0.0), dt=time_step(case), wall_level=2.0, voxel_size=1.0 / n, proj_iteration=10000)
    if "solver" in case:
        params["solver"] = flip.SOLVER_PLAIN if case["solver"] == "plain" else flip.SOLVER_MIXED
    if case.get("rk2"):
        params["advection"] = flip.ADVECT_RK2
    sim = flip.FlipSim(frame(case), (0.0, 0.0, 0.0), tuple(v / n for v in frame(case)), flip.default_params(**params))
    if case["scene"] == "tank":
        sim.set_colliders([(*tank_box(case), (0.0, 0.0, 0.0))], 3.0)
    return sim


def pinned(shape, dtype=torch.float32):
    return torch.empty(shape, dtype=dtype, pin_memory=True)


# ---- prepare and run -----------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "scan":
        gen = torch.Generator("cuda").manual_seed(seed)
        n = case["n"]
        state = {"case": case, "n": n, "lib": flip.load(),
                 "in": torch.randint(0, 20, (n,), generator=gen, device="cuda", dtype=torch.int32),
                 "out": torch.empty(n, device="cuda", dtype=torch.int32),
                 "total": torch.empty(1, device="cuda", dtype=torch.int32)}
        torch.cuda.synchronize()
        return state
    state = {"case": case, "sims": []}
    for k, c in enumerate(members(case)):
        pos, vel = particles(c, seed + 7919 * k)
        s = {"sim": make_sim(c), "pos": pinned(pos.shape), "vel": pinned(pos.shape), "n": pos.shape[0]}
        s["pos"].copy_(pos)
        s["vel"].copy_(vel)
        if kind in ("step", "batch"):
            s["pos_out"], s["vel_out"] = pinned(pos.shape), pinned(pos.shape)
        state["sims"].append(s)
    if kind in ("step", "batch"):
        run(state)  # simulations that have been running: their buffers have their size
        return state
    sim = s["sim"]
    sim.set_particles_ptr(s["pos"].data_ptr(), s["vel"].data_ptr(), s["n"])
    sim.run_stage(flip.STAGE_REBUILD)
    state["lib"], state["sim"] = flip.load(), sim
    cells = sim.frame_info()["ntiles"] * 512
    state["cells"] = cells
    for key in ("mass", "surf", "pres"):
        state[key] = pinned(cells)
    for key in ("velo", "comp"):
        state[key] = pinned((cells, 3))
    state["flag"] = pinned(cells, torch.uint8)
    if kind == "project":
        sim.run_stage(flip.STAGE_P2G)
    if kind in ("redistance", "vdb"):
        state["surf_in"] = pinned(cells)
        ijk = cell_coords(torch.from_numpy(sim.tiles()).cuda())
        state["surf_in"].copy_(surface_guess(case, seed, ijk))
        if kind == "vdb":
            sim.set_field(flip.FIELD_SURF, state["surf_in"].numpy())
            sim.set_field(flip.FIELD_VELO, velocity_guess(case, seed, ijk).cpu().numpy())
    run(state)
    return state


def distance(case, ijk):
    """Distance of the cell centres ijk (M, 3) to the scene's liquid, in voxels (negative inside)."""
    nx, ny, nz = frame(case)
    p = ijk.to(torch.float32) + 0.5
    d = torch.maximum(p[:, 0] - case["fx"] * nx, p[:, 1] - case["fy"] * ny)
    if case["sphere"]:
        c = torch.tensor([0.7 * nx, 0.8 * ny, 0.5 * nz], device="cuda")
        d = torch.minimum(d, (p - c).norm(dim=1) - case["sphere"] * min(nx, ny, nz))
    return p, d


def surface_guess(case, seed, ijk):
    """A stretched, noisy distance: what a particle splat hands to the redistancing."""
    gen = torch.Generator("cuda").manual_seed(seed)
    p, d = distance(case, ijk)
    par = torch.rand(3, generator=gen, device="cuda").tolist()
    d = d * (1.2 + 0.5 * par[0] * torch.sin(p[:, 0] * 0.21 + 6 * par[1]) * torch.sin(p[:, 2] * 0.17 + 6 * par[2]))
    d += 0.1 * (torch.rand(d.shape, generator=gen, device="cuda") - 0.5)
    return d.clamp(-0.5, 5.0)


def velocity_guess(case, seed, ijk):
    """A splatted velocity: noise on the cells within two voxels of the liquid, zero elsewhere."""
    gen = torch.Generator("cuda").manual_seed(seed + 1)
    _, d = distance(case, ijk)
    return torch.rand(len(d), 3, generator=gen, device="cuda").add_(0.1) * (d < 2.0).unsqueeze(1)


def fetch(state, which, key):
    out = state[key]
    st = state["lib"].bora_flip_get_field(state["sim"].h, which, ctypes.c_void_p(out.data_ptr()), out.numel() * out.element_size())
    if st != 0:
        raise RuntimeError(f"get_field: status {st}")
    return out


def run(state):
    kind = state["case"]["kind"]
    if kind == "scan":
        st = state["lib"].bora_scan_u32(*(ctypes.c_void_p(state[k].data_ptr()) for k in ("in", "out")), state["n"],
                                        ctypes.c_void_p(state["total"].data_ptr()),
                                        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st != 0:
            raise RuntimeError(f"scan: status {st}")
        return {"out": state["out"], "total": state["total"]}
    if kind in ("step", "batch"):
        return advance(state)
    sim = state["sim"]
    if kind == "grid":
        sim.run_stage(flip.STAGE_REBUILD)
        sim.run_stage(flip.STAGE_P2G)
        return {"mass": fetch(state, flip.FIELD_MASS, "mass"), "count": fetch(state, flip.FIELD_SURF, "surf"),
                "velo": fetch(state, flip.FIELD_VELO, "velo"), "flag": fetch(state, flip.FIELD_FLAG, "flag")}
    if kind == "project":
        sim.run_stage(flip.STAGE_BUILD_SYSTEM)
        sim.run_stage(flip.STAGE_SOLVE)
        sim.run_stage(flip.STAGE_UPDATE_VELOCITY)
        return {"pres": fetch(state, flip.FIELD_PRES, "pres"), "comp": fetch(state, flip.FIELD_COMP, "comp")}
    if kind == "splat":
        sim.run_post_stage(flip.POST_SPLAT)
        return {"surf": fetch(state, flip.FIELD_SURF, "surf"), "weight": fetch(state, flip.FIELD_PRES, "pres"),
                "velo": fetch(state, flip.FIELD_VELO, "velo")}
    if kind == "redistance":
        sim.set_field(flip.FIELD_SURF, state["surf_in"].numpy())
        sim.run_post_stage(flip.POST_REDISTANCE)
        return {"surf": fetch(state, flip.FIELD_SURF, "surf")}
    surface, velocity = sim.export_vdb(flip.VDB_SURFACE), sim.export_vdb(flip.VDB_VELOCITY)
    return [{"origins": d["origins"], "masks": d["masks"].view(np.int64), "values": d["values"]} for d in (surface, velocity)]


def advance(state):
    sims = state["sims"]
    for s in sims:
        s["sim"].set_particles_ptr(s["pos"].data_ptr(), s["vel"].data_ptr(), s["n"])
    if state["case"]["kind"] == "batch":
        flip.step_batch([s["sim"] for s in sims], time_step(members(state["case"])[-1]))
    else:
        sims[0]["sim"].step(time_step(state["case"]))
    out = []
    for s in sims:
        n = s["sim"].get_particles_ptr(s["pos_out"].data_ptr(), s["vel_out"].data_ptr(), s["n"])
        out += [s["pos_out"][:n], s["vel_out"][:n]]
    return out


def work(case):
    """Bytes: the caller's inputs once in and its outputs once out (and, where the particles stay on
    the device, their one read). Flops: the particles' transfers to and from the grid (8 corners, 4
    and 6 values) and one application of the 7-point operator per fluid cell."""
    kind = case["kind"]
    if kind == "scan":
        return {"bytes": 8.0 * case["n"], "flops": float(case["n"])}
    cells = 0
    for c in members(case):
        nx, ny, nz = frame(c)
        if c["scene"] == "tank":
            cells += nx * nz * c["depth"] + 0.04 * nx * nz * (0.3 * ny - c["depth"])
        else:
            cells += c["fx"] * nx * c["fy"] * ny * nz + 4.19 * c["sphere"] ** 3 * nx * ny * nz
    n = cells * PPC
    if kind in ("step", "batch"):
        return {"bytes": 48.0 * n, "flops": 400.0 * n + 40.0 * cells}
    if kind == "grid":
        return {"bytes": 24.0 * n + 21.0 * cells, "flops": 100.0 * n}
    if kind == "project":
        return {"bytes": (13.0 + 16.0) * cells, "flops": 40.0 * cells}
    if kind == "splat":
        return {"bytes": 24.0 * n + 20.0 * cells, "flops": 27 * 20.0 * n}
    if kind == "redistance":
        return {"bytes": 8.0 * cells, "flops": 80 * 50.0 * cells}
    return {"bytes": 32.0 * cells, "flops": 4.0 * cells}


# ---- the same in 64 bits --------------------------------------------------------------------

def exact(case, seed):
    kind = case["kind"]
    if kind in ("scan", "vdb"):
        return None  # whole numbers; copies scaled by one factor
    if kind in ("step", "batch"):
        out = []
        dt = time_step(members(case)[-1])
        for k, c in enumerate(members(case)):
            r = exact_step(c, *particles(c, seed + 7919 * k), dt)
            if r is None:
                return None
            out += r
        return out
    pos, vel = particles(case, seed)
    tiles = active_tiles(case, pos)
    ijk = cell_coords(tiles)
    if kind == "redistance":
        return {"surf": exact_redistance(case, tiles, ijk, surface_guess(case, seed, ijk)).cpu()}
    if kind == "splat":
        surf, weight, velo = exact_splat(case, pos, vel)
        return {"surf": pick(surf, ijk, 5.0), "weight": pick(weight, ijk, 0.0), "velo": pick(velo, ijk, 0.0)}
    G = exact_grid(case, pos, vel)
    if kind == "grid":
        flag = pick((G["mass"] > 0).to(torch.uint8) * 4, ijk, 255)
        return {"mass": pick(G["mass"], ijk, 0.0), "count": pick(G["count"], ijk, 0.0), "velo": pick(G["velo"], ijk, 0.0),
                "flag": flag}
    if G["mass"].numel() > EXACT_CELLS:
        return None
    pres, comp = exact_project(case, G)
    return {"pres": pick(pres, ijk, 0.0), "comp": pick(comp, ijk, 0.0)}


def active_tiles(case, pos):
    """Tile coordinates (T, 3) of the 8^3 tiles within one tile of a particle, x fastest."""
    tx, ty, tz = ((f + 7) // 8 for f in frame(case))
    t = (pos.to(torch.int64) // 8).clamp(min=0)
    lim = torch.tensor([tx - 1, ty - 1, tz - 1], device="cuda")
    t = torch.minimum(t, lim)
    occ = torch.zeros(tz, ty, tx, device="cuda")
    occ[t[:, 2], t[:, 1], t[:, 0]] = 1
    act = torch.nn.functional.max_pool3d(occ[None, None], 3, stride=1, padding=1)[0, 0]
    return act.nonzero().flip(1)


def cell_coords(tiles):
    """Cell coordinates (T * 512, 3) in the fields' storage order."""
    l = torch.arange(512, device="cuda")
    loc = torch.stack([l & 7, (l >> 3) & 7, l >> 6], 1)
    return (tiles.reshape(-1, 1, 3) * 8 + loc).reshape(-1, 3)


def pick(dense, ijk, beyond):
    """The values of a dense (nz, ny, nx[, 3]) field at the storage order's cells."""
    nz, ny, nx = dense.shape[:3]
    inside = (ijk[:, 0] < nx) & (ijk[:, 1] < ny) & (ijk[:, 2] < nz)
    c = ijk.clamp(max=torch.tensor([nx - 1, ny - 1, nz - 1], device="cuda"))
    v = dense[c[:, 2], c[:, 1], c[:, 0]]
    v[~inside] = beyond
    return v.cpu()


def exact_grid(case, pos, vel):
    """P2G (Rasterization.cu:122-229) on the dense grid, cropped in y to the layers that can hold fluid."""
    nx, ny, nz = frame(case)
    _, top = filled(case)
    ny = min(ny, top + 4) if case["scene"] == "tank" else ny
    base = (pos - 0.5).to(torch.int64).clamp(min=0)
    mass = torch.zeros(nz * ny * nx, dtype=torch.float64, device="cuda")
    count = torch.zeros_like(mass)
    mom = [torch.zeros_like(mass) for _ in range(3)]
    ext = (nx, ny, nz)
    for o in range(8):
        c = [base[:, a] + ((o >> a) & 1) for a in range(3)]
        ok = (c[0] < nx) & (c[1] < ny) & (c[2] < nz)
        lin = torch.where(ok, (c[2] * ny + c[1]) * nx + c[0], 0)
        w = torch.ones(pos.shape[0], dtype=torch.float64, device="cuda")
        for a in range(3):
            w *= (1.0 - (pos[:, a].double() - (c[a].double() + 0.5)).abs()).clamp(min=0.0)
        w += float(np.float32(1e-5))
        w *= ok
        mass.index_add_(0, lin, w)
        count.index_add_(0, lin, ok.double())
        for a in range(3):
            mom[a].index_add_(0, lin, w * vel[:, a].double())
        del c, ok, lin, w
    shape = (nz, ny, nx)
    velo = torch.stack([torch.where(mass > 0, m / mass.clamp(min=1e-300), m).view(shape) for m in mom], 3)
    return {"mass": mass.view(shape), "count": count.view(shape), "velo": velo, "ext": ext}


def solid_cells(case, shape):
    """Cells whose centre lies in the tank's obstacle."""
    nz, ny, nx = shape
    if case["scene"] != "tank":
        return torch.zeros(shape, dtype=torch.bool, device="cuda")
    lo, hi = tank_box(case)
    m = torch.ones(shape, dtype=torch.bool, device="cuda")
    for a, (n, view) in enumerate(((nx, (1, 1, nx)), (ny, (1, ny, 1)), (nz, (nz, 1, 1)))):
        x = (torch.arange(n, device="cuda") + 0.5).view(view)
        m &= (x > lo[a]) & (x < hi[a])
    return m


def neighbours(f, edge_lo, edge_hi, axis):
    """f at the cells below and above along an axis of (z, y, x); edge_lo / edge_hi fill the grid's faces."""
    lo, hi = torch.empty_like(f), torch.empty_like(f)
    n = f.shape[axis]
    lo.narrow(axis, 1, n - 1).copy_(f.narrow(axis, 0, n - 1))
    hi.narrow(axis, 0, n - 1).copy_(f.narrow(axis, 1, n - 1))
    lo.narrow(axis, 0, 1).copy_(edge_lo if torch.is_tensor(edge_lo) else torch.full_like(lo.narrow(axis, 0, 1), edge_lo))
    hi.narrow(axis, n - 1, 1).copy_(edge_hi if torch.is_tensor(edge_hi) else torch.full_like(hi.narrow(axis, n - 1, 1), edge_hi))
    return lo, hi


AIR, SOLID, WALL, FLUID = 0, 1, 2, 4


def exact_project(case, G):
    """FluidProjection (FluidProjection.cu:165-381) with solid walls on every face: the pressure by conjugate
    gradients to 1e-12, then the projected velocity. A cropped top face lies in air and counts as such."""
    mass, velo = G["mass"], G["velo"]
    cropped = mass.shape[1] < frame(case)[1]
    fluid = mass > 0
    flag = torch.where(fluid, FLUID, torch.where(solid_cells(case, mass.shape), SOLID, AIR)).to(torch.int8)
    axis_of = (2, 1, 0)  # x, y, z in (z, y, x) storage
    diag = torch.full_like(mass, 6.0)
    div = torch.zeros_like(mass)
    types = []
    for a in range(3):
        ax = axis_of[a]
        t0, t1 = neighbours(flag, WALL, AIR if a == 1 and cropped else WALL, ax)
        types.append((t0, t1))
        v = velo[..., a]
        n = v.shape[ax]
        e0 = 2 * v.narrow(ax, 0, 1) - v.narrow(ax, 1, 1)
        e1 = 2 * v.narrow(ax, n - 1, 1) - v.narrow(ax, n - 2, 1)
        lo, hi = neighbours(v, e0, e1, ax)
        v0 = torch.where(t0 == AIR, 2 * v - hi, torch.where(t0 == WALL, v.abs(), lo))
        v1 = torch.where(t1 == AIR, 2 * v - lo, torch.where(t1 == WALL, -v.abs(), hi))
        div += (v1 - v0) * 0.5
        for t in (t0, t1):
            diag += (t == AIR).double() - ((t == SOLID) | (t == WALL)).double()
    b = torch.where(fluid, -div, 0.0)
    p = conjugate_gradients(diag, fluid, b)
    # air cells next to fluid take the mean of their fluid neighbours' pressure
    total, cnt = torch.zeros_like(p), torch.zeros_like(p)
    for a in range(3):
        lo, hi = neighbours(p, 0.0, 0.0, axis_of[a])
        for t, q in zip(types[a], (lo, hi)):
            total += torch.where(t == FLUID, q, 0.0)
            cnt += (t == FLUID).double()
    p = torch.where((flag == AIR) & (cnt > 0), total / cnt.clamp(min=1.0), p)
    comp = velo.clone()
    for a in range(3):
        ax = axis_of[a]
        n = p.shape[ax]
        e0 = 2 * p.narrow(ax, 0, 1) - p.narrow(ax, 1, 1)
        e1 = 2 * p.narrow(ax, n - 1, 1) - p.narrow(ax, n - 2, 1)
        lo, hi = neighbours(p, e0, e1, ax)
        t0, t1 = ((t == SOLID) | (t == WALL) for t in types[a])
        p0 = torch.where(t0, 2 * p - hi, torch.where(types[a][0] == AIR, -lo, lo))
        p1 = torch.where(t1, 2 * p - lo, torch.where(types[a][1] == AIR, -hi, hi))
        comp[..., a] -= torch.where(fluid, (p1 - p0) * 0.5, 0.0)
    return p, comp


def conjugate_gradients(diag, fluid, b):
    x, r = torch.zeros_like(b), b.clone()
    inv = torch.where(fluid, 1.0 / diag.clamp(min=1.0), 0.0)
    z = inv * r
    d = z.clone()
    rz = (r * z).sum()
    stop = 1e-12 * float(b.norm())
    for it in range(20000):
        q = diag * d
        for ax in range(3):
            n = d.shape[ax] - 1
            q.narrow(ax, 1, n).sub_(d.narrow(ax, 0, n))
            q.narrow(ax, 0, n).sub_(d.narrow(ax, 1, n))
        q *= fluid
        alpha = rz / (d * q).sum().clamp(min=1e-300)
        x += alpha * d
        r -= alpha * q
        if it % 25 == 24 and float(r.norm()) <= stop:
            break
        z = inv * r
        new = (r * z).sum()
        d.mul_(new / rz.clamp(min=1e-300)).add_(z)
        rz = new
    return x


def lerp_at(fields, pos):
    """Trilinear values of (nz, ny, nx, C) fields at points, cell-centred and clamped (SparseField.h:150-173)."""
    nz, ny, nx, _ = fields.shape
    c, f = [], []
    for a, n in enumerate((nx, ny, nz)):
        i = (pos[:, a] - 0.5).to(torch.int64).clamp(0, n - 2)
        c.append(i)
        f.append((pos[:, a].double() - (i.double() + 0.5)).clamp(0.0, 1.0).unsqueeze(1))
    out = 0.0
    for o in range(8):
        w = 1.0
        for a in range(3):
            w = w * (f[a] if (o >> a) & 1 else 1.0 - f[a])
        out = out + w * fields[c[2] + (o >> 2), c[1] + ((o >> 1) & 1), c[0] + (o & 1)]
    return out


def exact_step(case, pos, vel, dt):
    """One advanceOneStep (FLIPMethod.cu:54-298) with solid walls; particles in the sort's order."""
    nx, ny, nz = frame(case)
    G = exact_grid(case, pos, vel)
    if G["mass"].numel() > EXACT_CELLS:
        return None
    _, comp = exact_project(case, G)
    velo = G["velo"]
    tx, ty = (nx + 7) // 8, (ny + 7) // 8
    base = (pos - 0.5).to(torch.int64).clamp(min=0)
    t, l = base >> 3, base & 7
    key = ((t[:, 2] * ty + t[:, 1]) * tx + t[:, 0]) * 512 + l[:, 0] + 8 * l[:, 1] + 64 * l[:, 2]
    order = torch.sort(key, stable=True)[1]
    del base, t, l, key
    new_pos, new_vel = [], []
    fields = torch.cat([comp, velo], 3)
    grav = -9.8 * float(max(frame(case)))
    for part in order.split(4_000_000):
        p, v = pos[part], vel[part].double()
        s = lerp_at(fields, p)
        gn, go = s[:, :3], s[:, 3:]
        v = (v + gn - go) * float(np.float32(0.95)) + gn * float(np.float32(0.05))
        p = p.double()
        iters = 1 + (v.norm(dim=1) * dt * 1.5).to(torch.int64).clamp(max=1)
        sub = (dt / iters.double()).unsqueeze(1)
        lim = torch.tensor([nx, ny, nz], dtype=torch.float64, device="cuda")
        for it in range(2):
            live = (iters > it).unsqueeze(1)
            if case["rk2"]:
                k1 = lerp_at(comp, p)
                q = p + lerp_at(comp, p + k1 * (0.5 * sub)) * sub
            else:
                q = p + v * sub
            below, above = q < 0, q > lim
            w = torch.where((below & (v < 0)) | (above & (v > 0)), 0.0, v)
            q = torch.minimum(q.clamp(min=0.0), lim)
            p, v = torch.where(live, q, p), torch.where(live, w, v)
        v[:, 1] += grav * dt
        new_pos.append(p.cpu())
        new_vel.append(v.cpu())
    return [torch.cat(new_pos), torch.cat(new_vel)]


def exact_splat(case, pos, vel):
    """ParticlesToSurfaceAndVelocity (Rasterization.cu:311-398), influence 1.5, droplet 0.5."""
    nx, ny, nz = frame(case)
    shape = (nz, ny, nx)
    acc = torch.zeros(nz * ny * nx, 7, dtype=torch.float64, device="cuda")
    data = torch.cat([torch.ones_like(pos[:, :1]), pos, vel], 1).double()
    base = pos.to(torch.int64)
    for o in range(27):
        c = base + torch.tensor([o % 3 - 1, o // 3 % 3 - 1, o // 9 - 1], device="cuda")
        ok = ((c >= 0) & (c < torch.tensor([nx, ny, nz], device="cuda"))).all(1)
        d2 = ((pos.double() - (c.double() + 0.5)) ** 2).sum(1)
        w = (1.0 - d2 / 2.25).clamp(min=0.0) ** 3 * ok
        lin = torch.where(ok, (c[:, 2] * ny + c[:, 1]) * nx + c[:, 0], 0)
        acc.index_add_(0, lin, data * w.unsqueeze(1))
    weight = acc[:, 0]
    some = weight > 1e-30
    mean = acc[:, 1:] / weight.clamp(min=1e-30).unsqueeze(1)
    k, j, i = torch.meshgrid(*(torch.arange(n, device="cuda") + 0.5 for n in shape), indexing="ij")
    centre = torch.stack([i, j, k], 3).view(-1, 3).double()
    surf = torch.where(some, (mean[:, :3] - centre).norm(dim=1) - 0.5, 5.0)
    velo = torch.where(some.unsqueeze(1), mean[:, 3:], 0.0)
    return surf.view(shape), weight.view(shape), velo.view(*shape, 3)


def exact_redistance(case, tiles, ijk, surf):
    """80 steps of ReinitializeSurface (Rasterization.cu:400-486) on the active tiles' cells."""
    nx, ny, nz = frame(case)
    inside = (ijk[:, 0] < nx) & (ijk[:, 1] < ny) & (ijk[:, 2] < nz)
    c = ijk[inside]
    f = torch.full((nz, ny, nx), SURF_BACKGROUND, dtype=torch.float64, device="cuda")
    act = torch.zeros((nz, ny, nx), dtype=torch.bool, device="cuda")
    f[c[:, 2], c[:, 1], c[:, 0]] = surf.double()[inside]
    act[c[:, 2], c[:, 1], c[:, 0]] = True
    dt = float(np.float32(0.3))
    for _ in range(80):
        a, b = torch.zeros_like(f), torch.zeros_like(f)
        for ax in range(3):
            n = f.shape[ax]
            lo, hi = neighbours(f, 2 * f.narrow(ax, 0, 1) - f.narrow(ax, 1, 1),
                                2 * f.narrow(ax, n - 1, 1) - f.narrow(ax, n - 2, 1), ax)
            d0, d1 = f - lo, hi - f
            a += d0.clamp(min=0) ** 2 + d1.clamp(max=0) ** 2
            b += d0.clamp(max=0) ** 2 + d1.clamp(min=0) ** 2
        sign = f / (f * f + 1).sqrt()
        step_ = dt * sign.clamp(min=0) * (a.sqrt() - 1) + dt * sign.clamp(max=0) * (b.sqrt() - 1)
        f = torch.where(act, f - step_, f)
    out = surf.double().clone()
    out[inside] = f[c[:, 2], c[:, 1], c[:, 0]]
    return out
