"""Performance cases of the coarse-grid field step, through the package's
public Python entry points (`tpt_field`, `voxel3d`).

A case is a dict of plain values. `kind` selects the entry points:

  air      `step_air_gpu` on one canvas
  frame    what an engine calls per frame of one canvas with Newtonian gravity
           on: `step_air_gpu` (with the HotAir particle map) + `step_gravity`
  gravity  `GravityFft.solve` on one canvas
  gravtick `GravityFft.step`: wells, solve, force on the particles, mass build
  batch    `Batch.step` of many sandboxes, results read to pinned host memory
  voxel    the 3-D sandbox's `field_step` and `gravity_gather`

`listed` has the named cases, `draw` makes others of the same ranges,
`prepare` / `run` are a user's program before and in the loop, `work` counts
what a pass cannot do without and `exact` computes float64 results with plain
torch operations.
"""
import math
import os
import sys

import numpy as np
import torch

# The package's folder is not an importable name: its modules are imported
# from it, relative to the working folder (the repository's root).
_PKG = os.path.join(os.getcwd(), "the-powder-toy-rust-wgpu_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import tpt_field as tf  # noqa: E402
import voxel3d as V  # noqa: E402
import workloads as W  # noqa: E402

M_GRAV = 6.673e-1
F32_GRAV, BF16_GRAV = "fp32", "split_bf16"
PRECISION = {F32_GRAV: tf.PRECISION_FP32, BF16_GRAV: tf.PRECISION_SPLIT_BF16}
N_ELEMENTS = 192


# ------------------------------------------------------------------ cases --

def listed():
    return [
        # The smallest canvas SimulationConfig.new allows (64x64 px): a call
        # is launches and latency.
        {"name": "air_smallest", "kind": "air", "x": 16, "y": 16, "options": 0},
        # One frame of the default 612x384 canvas with gravity and particles
        # that heat the air: what every interactive user runs.
        {"name": "frame_default", "kind": "frame", "x": 153, "y": 96, "options": 1},
        # A 1600x900 canvas with every option in use: fans, powered walls,
        # radial gravity, legacy convection, odd sides.
        {"name": "air_canvas", "kind": "air", "x": 401, "y": 225, "options": 2},
        # The largest canvas the library takes (8192x8192 px).
        {"name": "air_largest", "kind": "air", "x": 2048, "y": 2048, "options": 1},
        # Gravity of a 1600x900 canvas from the engine's fixed-point mass.
        {"name": "grav_f32", "kind": "gravity", "x": 400, "y": 225, "precision": F32_GRAV, "f32_mass": False},
        # A canvas longer than the 2048 px the reference's UI offers.
        {"name": "grav_f32_long", "kind": "gravity", "x": 1200, "y": 701, "precision": F32_GRAV, "f32_mass": False},
        # The gravity-only workload: 512x512 cells, clustered f32 mass, on the
        # tensor cores.
        {"name": "grav_bf16", "kind": "gravity", "x": 512, "y": 512, "precision": BF16_GRAV, "f32_mass": True},
        # A gravity tick with the default canvas's particle slots half full.
        {"name": "grav_particles", "kind": "gravtick", "x": 153, "y": 96, "slots": 117500, "precision": F32_GRAV},
        # Many sandboxes of many sizes, all FP32: 256 grids, sides log-uniform
        # in 32..512.
        {"name": "batch_mixed_f32", "kind": "batch", "big": 0, "tail": 256, "ticks": 40, "precision": F32_GRAV,
         "log_uniform": True, "tune": False},
        # The headline batch: 64 canvases of 1600x900 px and 64 heavy-tailed
        # ones, split-BF16 gravity, tuned once as the benchmark does.
        {"name": "batch_headline", "kind": "batch", "big": 64, "tail": 64, "ticks": 100, "precision": BF16_GRAV,
         "log_uniform": False, "tune": True},
        # One 3-D world with every brick active, one tick.
        {"name": "voxel_one", "kind": "voxel", "worlds": 1, "active": 1.0, "iterations": 12},
        # A server's eight 3-D worlds in one call, a third of the bricks active.
        {"name": "voxel_eight", "kind": "voxel", "worlds": 8, "active": 0.3, "iterations": 12},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["air", "frame", "gravity", "gravity", "gravtick", "batch", "voxel"])
    if kind in ("air", "frame"):
        return {"kind": kind, "x": _log_int(rng, 16, 2048), "y": _log_int(rng, 16, 2048), "options": rng.randrange(3)}
    if kind == "gravity":
        prec = rng.choice([F32_GRAV, BF16_GRAV])
        top = 1500 if prec == F32_GRAV else 700
        return {"kind": kind, "x": _log_int(rng, 16, top), "y": _log_int(rng, 16, top), "precision": prec,
                "f32_mass": rng.random() < 0.5}
    if kind == "gravtick":
        return {"kind": kind, "x": _log_int(rng, 16, 512), "y": _log_int(rng, 16, 512),
                "slots": _log_int(rng, 1000, 1000000), "precision": rng.choice([F32_GRAV, BF16_GRAV])}
    if kind == "batch":
        return {"kind": kind, "big": rng.choice([0, 1, 5, 12, 24]), "tail": _log_int(rng, 2, 96),
                "ticks": rng.randrange(1, 61), "precision": rng.choice([F32_GRAV, BF16_GRAV]),
                "log_uniform": rng.random() < 0.5, "tune": False}
    return {"kind": kind, "worlds": _log_int(rng, 1, 8), "active": round(rng.uniform(0.02, 1.0), 3),
            "iterations": rng.choice([4, 12, 13, 20])}


# ----------------------------------------------------------------- inputs --

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + 17)
    return g


def _uniform(g, n, lo, hi, dtype=torch.float32):
    return lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=dtype)


def _ints(g, n, lo, hi):
    return torch.randint(lo, hi, (n,) if isinstance(n, int) else n, generator=g, device="cuda", dtype=torch.int64)


def _blobs(g, X, Y, amplitude, count=8):
    """A sum of `count` Gaussians (sigma 3..12 cells), (Y, X)."""
    cx, cy = _uniform(g, count, 1, max(X - 1, 2)), _uniform(g, count, 1, max(Y - 1, 2))
    sg, amp = _uniform(g, count, 3, 12), _uniform(g, count, -amplitude, amplitude)
    xs, ys = torch.arange(X, device="cuda"), torch.arange(Y, device="cuda")
    ex = torch.exp(-((xs[None, :] - cx[:, None]) ** 2) / (2 * sg[:, None] ** 2))
    ey = torch.exp(-((ys[:, None] - cy[None, :]) ** 2) / (2 * sg[None, :] ** 2))
    # an exact order of additions: the inputs do not depend on a GEMM's split
    out = torch.zeros(Y, X, device="cuda")
    for k in range(count):
        out += amp[k] * ey[:, k, None] * ex[k, None, :]
    return out


def _walls(g, X, Y, options):
    """Wall ids and emap: a border ring and 5% of the interior are WALL; with
    options 2 powered e-walls, fans and a ring of gravity walls too."""
    wall = torch.zeros(Y, X, dtype=torch.int64, device="cuda")
    u = _uniform(g, (Y, X), 0, 1)
    wall[u < 0.05] = W.WL_WALL
    emap = torch.zeros_like(wall)
    gmask = torch.ones(Y, X, dtype=torch.bool, device="cuda")
    if options == 2:
        wall[(u >= 0.05) & (u < 0.06)] = W.WL_EWALL
        wall[(u >= 0.06) & (u < 0.07)] = W.WL_FAN
        emap = torch.where(wall == W.WL_EWALL, _ints(g, (Y, X), 0, 4), emap)
    wall[0, :] = wall[-1, :] = W.WL_WALL
    wall[:, 0] = wall[:, -1] = W.WL_WALL
    if options == 2 and X >= 16 and Y >= 16:  # a closed ring of gravity walls: masked inside
        x0, y0 = X // 4, Y // 4
        wall[y0:y0 + 7, x0:x0 + 7] = W.WL_GRAV
        wall[y0 + 1:y0 + 6, x0 + 1:x0 + 6] = 0
        gmask[y0:y0 + 7, x0:x0 + 7] = False
    return wall, emap, gmask


def _mass(g, n, density, lo=0.0, hi=1.0):
    m = torch.where(_uniform(g, n, 0, 1) < density, _uniform(g, n, lo, hi), torch.zeros(n, device="cuda"))
    return torch.floor(m.double() * 65536 + 0.5).to(torch.int32)


def _host(t, dtype):
    return t.reshape(-1).to(torch.int64 if dtype == np.uint32 else t.dtype).cpu().numpy().astype(dtype)


def _instance(g, X, Y, options):
    """A sandbox in mid-run: blob pressure and velocity, air at 20..30 C.
    options: 0 the default configuration (no ambient heat), 1 with ambient
    heat, 2 with every wall kind, radial gravity and legacy convection too."""
    wall, emap, gmask = _walls(g, X, Y, options)
    pv = torch.clamp(_blobs(g, X, Y, 200.0), -256, 256)
    vx, vy = torch.clamp(_blobs(g, X, Y, 6.0), -256, 256), torch.clamp(_blobs(g, X, Y, 6.0), -256, 256)
    hv = _uniform(g, (Y, X), 273.15 + 20, 273.15 + 30)
    fan = wall == W.WL_FAN
    fvx = torch.where(fan, _uniform(g, (Y, X), -2, 2), torch.zeros_like(pv))
    fvy = torch.where(fan, _uniform(g, (Y, X), -2, 2), torch.zeros_like(pv))
    mass = _mass(g, X * Y, 0.02)
    wall_h, emap_h = _host(wall, np.uint32), _host(emap, np.uint32)
    bair, bairh = W.wall_masks(wall_h, emap_h)
    zero = np.zeros(X * Y, np.uint32)
    cfg = W.AirConfig(aheat_enable=int(options != 0))
    if options == 2:
        cfg = W.AirConfig(convection_mode=1, gravity_mode=2, edge_pressure=0.5, edge_vx=0.25, edge_vy=-0.125)
    gm = np.where(_host(gmask, np.uint32) != 0, np.uint32(0xFFFFFFFF), np.uint32(0))
    return W.Instance(X, Y, cfg, pv=_host(pv, np.float32), vx=_host(vx, np.float32), vy=_host(vy, np.float32),
                      hv=_host(hv, np.float32), wall=wall_h, emap=emap_h, bair=bair, bairh=bairh, eair=zero,
                      eairh=zero.copy(), fan_vx=_host(fvx, np.float32), fan_vy=_host(fvy, np.float32),
                      mass_fx=_host(mass, np.int32), gmask=gm)


def _particle_map(g, X, Y):
    """A pixel map with a fifth of the pixels occupied, and an element table
    in which some elements heat or cool the air (gases among them)."""
    n = X * Y * 16
    ty = _ints(g, n, 1, N_ELEMENTS)
    ident = torch.arange(n, device="cuda") << 9
    pmap = torch.where(_uniform(g, n, 0, 1) < 0.2, ty | ident, torch.zeros_like(ty))
    hot = torch.zeros(N_ELEMENTS, device="cuda")
    some = _ints(g, N_ELEMENTS, 0, 8) == 0
    some[10] = some[97] = True
    hot = torch.where(some, _uniform(g, N_ELEMENTS, -0.0001, 0.001), hot)
    props = torch.zeros(N_ELEMENTS, 32, dtype=torch.int32, device="cuda")
    props[:, 11] = hot.view(torch.int32)
    return (pmap & 0x7FFFFFFF).to(torch.int32), props.reshape(-1)


def _shapes(case):
    """The batch's grid sizes: `big` canvases of 400x225 cells, then `tail`
    log-uniform or Pareto(1.5) ones, as in the two batched workloads. The
    sizes belong to the case, not to the seed."""
    st = W.Stream(W.CONFIG_SEED_BASE + (4 if case["log_uniform"] else 5))
    n = case["tail"]
    u, v = st.uniform(0.0, 1.0, n), st.uniform(0.0, 1.0, n)
    if case["log_uniform"]:
        w, h = [np.rint(32 * np.exp(a * math.log(16))).astype(int) for a in (u, v)]
    else:
        w, h = [np.clip(np.floor(32.0 * (1.0 - a) ** (-1.0 / 1.5)), 32, 512).astype(int) for a in (u, v)]
    return [(400, 225)] * case["big"] + [(int(a), int(b)) for a, b in zip(w, h)]


def _instances(case, seed):
    g = _gen(seed)
    return [_instance(g, X, Y, 2 if i % 16 == 7 else 1) for i, (X, Y) in enumerate(_shapes(case))]


def _gravity_inputs(case, seed):
    g, X, Y = _gen(seed), case["x"], case["y"]
    wall, _, gmask = _walls(g, X, Y, 2)
    if case["f32_mass"]:
        mass = torch.abs(_blobs(g, X, Y, 5.0, 50)).reshape(-1)
        mass = mass + torch.where(_uniform(g, X * Y, 0, 1) < 0.01, _uniform(g, X * Y, 0, 1), torch.zeros_like(mass))
    else:
        mass = _mass(g, X * Y, 0.03)
    return mass.contiguous(), gmask.reshape(-1)


def _tick_inputs(case, seed):
    """Particle slots (a quarter empty, a tenth gravity elements), the element
    table and the gravity grids of a sandbox in mid-run."""
    g, X, Y, n = _gen(seed), case["x"], case["y"], case["slots"]
    ty = _ints(g, n, 1, N_ELEMENTS)
    u = _uniform(g, n, 0, 1)
    ty = torch.where(u < 0.1, _ints(g, n, 39, 44), ty)
    ty = torch.where(u > 0.75, torch.zeros_like(ty), ty)
    parts = {"ty": ty, "x": _uniform(g, n, 0, 4 * X - 1), "y": _uniform(g, n, 0, 4 * Y - 1),
             "vx": _uniform(g, n, -4, 4), "vy": _uniform(g, n, -4, 4), "life": _ints(g, n, 0, 40),
             "tmp": _ints(g, n, -300, 300), "temp": _uniform(g, n, 250, 1200),
             "flags": torch.where(_uniform(g, n, 0, 1) < 0.05, _ints(g, n, 0, 4) * 8, torch.zeros_like(ty))}
    parts = {k: v if v.dtype == torch.float32 else v.to(torch.int32) for k, v in parts.items()}
    lut = torch.zeros(N_ELEMENTS, 12, dtype=torch.int32, device="cuda")
    lut[:, 0] = torch.where(_ints(g, N_ELEMENTS, 0, 3) == 0, 4, 0)
    lut[:, 7] = _uniform(g, N_ELEMENTS, 0.5, 1.0).view(torch.int32)
    wall, _, gmask = _walls(g, X, Y, 2)
    wall = torch.where(_uniform(g, (Y, X), 0, 1) < 0.02, torch.full_like(wall, W.WL_STASIS), wall)
    cells = X * Y
    state = {"wall_bmap": wall.reshape(-1).to(torch.int32), "wall_emap": _ints(g, cells, 0, 16).to(torch.int32),
             "grav_mask": torch.where(gmask.reshape(-1), -1, 0).to(torch.int32),
             "mass": torch.zeros(cells, dtype=torch.int32, device="cuda"), "mass_prev": _mass(g, cells, 0.1, -1, 3),
             "tool_mass": torch.where(_uniform(g, cells, 0, 1) < 0.005, _uniform(g, cells, -5, 5),
                                      torch.zeros(cells, device="cuda")),
             "override_mass": _ints(g, cells, -100000, 100000).to(torch.int32),
             "override_set": (_uniform(g, cells, 0, 1) < 0.002).to(torch.int32),
             "gx": torch.zeros(cells, device="cuda"), "gy": torch.zeros(cells, device="cuda")}
    return parts, lut.reshape(-1), state


AIR_FIELDS = ("vx", "vy", "vz", "p", "p_tmp", "t", "solid", "pv")
GRAV_FIELDS = ("grav_mass", "grav_potential", "grav_potential_tmp", "grav_force_x", "grav_force_y", "grav_force_z")


def _worlds(case, seed):
    """3-D worlds in mid-run and, per field, the tensor whose rows are the
    worlds' grids: 40% of the voxels are occupied, `active` of the bricks
    listed in random order."""
    g, count, nv, nc = _gen(seed), case["worlds"], W.VOX_VOXELS, W.VOX_CELLS
    fields = {k: torch.zeros(count, nc, dtype=torch.int32 if k in ("pv", "grav_mass") else torch.float32, device="cuda")
              for k in AIR_FIELDS + GRAV_FIELDS}
    kinds = torch.tensor([1, 5, 27, 39, 40, 41, 42, 43, 100, 255], device="cuda")
    n = max(1, int(round(case["active"] * W.VOX_BRICKS)))
    worlds = []
    for i in range(count):
        b, air = V.Voxel3dBuffers.__new__(V.Voxel3dBuffers), V.AirState.__new__(V.AirState)
        ty = torch.where(_uniform(g, nv, 0, 1) < 0.4, kinds[_ints(g, nv, 0, 10)], 0)
        b.voxel_a = (ty | (_ints(g, nv, 2000, 4000) << 8) | (_ints(g, nv, 0, 40) << 24)).to(torch.int32)
        b.aux_tmp = _ints(g, nv, -300, 300).to(torch.int32)
        b.sim_list = torch.zeros(W.VOX_BRICKS, dtype=torch.int32, device="cuda")
        b.sim_list[:n] = torch.randperm(W.VOX_BRICKS, generator=g, device="cuda")[:n].to(torch.int32)
        b.sim_count = torch.tensor([n, 1, 1], dtype=torch.int32, device="cuda")
        air.iterations = case["iterations"]
        for k in AIR_FIELDS:
            setattr(air, k, fields[k][i])
        for k in GRAV_FIELDS:
            setattr(b, k, fields[k][i])
        b.grav_mass.copy_(torch.where(_uniform(g, nc, 0, 1) < 0.02, _ints(g, nc, -100000, 100000), 0))
        b.grav_potential.copy_(_uniform(g, nc, -50, 50))
        for k, lo, hi in (("vx", -8, 8), ("vy", -8, 8), ("vz", -8, 8), ("p", -2, 2), ("t", 250, 600)):
            getattr(air, k).copy_(_uniform(g, nc, lo, hi))
        air.pv.copy_(_ints(g, nc, -262144, 262145))
        worlds.append((b, air))
    return worlds, fields


# ------------------------------------------------------------ prepare, run --

def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("air", "frame"):
        g = _gen(seed)
        s["bufs"] = b = tf.SimBuffers.from_instance(_instance(g, case["x"], case["y"], case["options"]))
        if kind == "frame":
            b.config.newton_grav = True
            b.pmap, b.elem_props = _particle_map(g, case["x"], case["y"])
            s["solver"] = tf.GravityFft(tf.PRECISION_FP32)
            s["solver"]._ensure(case["x"], case["y"])
    elif kind == "gravity":
        mass, gmask = _gravity_inputs(case, seed)
        s["bufs"] = b = tf.SimBuffers(tf.SimulationConfig(xres=4 * case["x"], yres=4 * case["y"], newton_grav=True))
        b.grav_mask.copy_(torch.where(gmask, -1, 0))
        b.grav_mask_dirty = False
        s["mass"] = mass
        s["solver"] = tf.GravityFft(PRECISION[case["precision"]])
        s["solver"]._ensure(case["x"], case["y"])
    elif kind == "gravtick":
        s["parts"], s["lut"], s["state"] = _tick_inputs(case, seed)
        s["solver"] = tf.GravityFft(PRECISION[case["precision"]])
        s["solver"]._ensure(case["x"], case["y"])
    elif kind == "batch":
        s["batch"] = batch = tf.Batch(_instances(case, seed), PRECISION[case["precision"]])
        if case["tune"]:
            batch.tune()
        names = (("pv", tf.FIELD_PV), ("vx", tf.FIELD_VX), ("vy", tf.FIELD_VY), ("hv", tf.FIELD_HV),
                 ("gx", tf.FIELD_GX), ("gy", tf.FIELD_GY))
        s["out"] = {k: (f, torch.empty(batch.total_cells, pin_memory=True).numpy()) for k, f in names}
    else:
        s["plan"] = V.Plan()
        s["worlds"], s["fields"] = _worlds(case, seed)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("air", "frame"):
        b = s["bufs"]
        tf.step_air_gpu(b)
        out = {"pv": b.air_pv, "vx": b.air_vx, "vy": b.air_vy, "hv": b.air_hv, "block_air": b.block_air,
               "block_airh": b.block_airh, "emap": b.wall_emap}
        if kind == "frame":
            tf.step_gravity(b, s["solver"])
            out.update(gx=b.grav_fx, gy=b.grav_fy)
        return out
    if kind == "gravity":
        b = s["bufs"]
        s["solver"].solve(b, s["mass"])
        return {"gx": b.grav_fx, "gy": b.grav_fy}
    if kind == "gravtick":
        st, p = s["state"], s["parts"]
        s["solver"].step(st, p, s["lut"], N_ELEMENTS, 4 * case["x"], 4 * case["y"])
        return {"gx": st["gx"], "gy": st["gy"], "vx": p["vx"], "vy": p["vy"], "mass": st["mass"],
                "mass_prev": st["mass_prev"], "tool": st["tool_mass"]}
    if kind == "batch":
        s["batch"].step(case["ticks"])
        return {k: s["batch"].read_field(f, np.float32, out=a) for k, (f, a) in s["out"].items()}
    V.field_step(s["plan"], s["worlds"], case["iterations"])
    for b, _ in s["worlds"]:
        V.gravity_gather(s["plan"], b)
    return {k: v for k, v in s["fields"].items() if k != "grav_potential_tmp"}


# ------------------------------------------------------------------- work --

def _grav_work(cells):
    """A real linear convolution by FFT: one forward and two inverse real
    transforms of four times the cells, two spectrum products; mass and mask
    in, two fields out."""
    n = 4 * cells
    return 16 * cells, 3 * 2.5 * n * math.log2(max(n, 2)) + 12 * n


# Air, per cell and tick: pv, vx, vy, hv and two masks read and written, the
# wall id, emap and two element stamps read; about 200 operations.
AIR_BYTES, AIR_FLOPS = 64, 200


def work(case):
    kind = case["kind"]
    if kind in ("air", "frame", "gravity", "gravtick"):
        cells = case["x"] * case["y"]
    if kind == "air":
        return {"bytes": AIR_BYTES * cells, "flops": AIR_FLOPS * cells}
    if kind == "frame":  # and the 16 pixels of the particle map under a cell
        gb, gf = _grav_work(cells)
        return {"bytes": (AIR_BYTES + 64) * cells + gb, "flops": AIR_FLOPS * cells + gf}
    if kind == "gravity":
        gb, gf = _grav_work(cells)
        return {"bytes": gb, "flops": gf}
    if kind == "gravtick":  # a slot: type, position, velocity in and out, flags; a cell: walls, wells, overrides
        gb, gf = _grav_work(cells)
        return {"bytes": gb + 28 * case["slots"] + 28 * cells, "flops": gf + 12 * case["slots"]}
    if kind == "batch":
        shapes = _shapes(case)
        total = sum(X * Y for X, Y in shapes)
        grav = [_grav_work(X * Y) for X, Y in shapes]
        t = case["ticks"]
        return {"bytes": t * (AIR_BYTES * total + sum(b for b, _ in grav)),
                "flops": t * (AIR_FLOPS * total + sum(f for _, f in grav))}
    # per listed voxel: its word read by the two gathers; per cell: the air and
    # gravity state in and out; per sweep and cell about 10 operations
    vox = 512 * max(1, round(case["active"] * W.VOX_BRICKS))
    return {"bytes": case["worlds"] * (4 * vox + 80 * W.VOX_CELLS),
            "flops": case["worlds"] * W.VOX_CELLS * 10.0 * (case["iterations"] + V.GRAVITY_ITERATIONS + 8)}


# ------------------------------------------------------------------ exact --

D = torch.float64


def _shift(a, dx, dy):
    """b[y, x] = a[y + dy, x + dx], zero (or False) outside."""
    Y, X = a.shape
    b = torch.zeros_like(a)
    b[max(0, -dy):min(Y, Y - dy), max(0, -dx):min(X, X - dx)] = a[max(0, dy):min(Y, Y + dy), max(0, dx):min(X, X + dx)]
    return b


def _smooth(fields, open_, inner):
    """3x3 Gaussian means; a closed or rim neighbour counts as the centre."""
    taps = torch.tensor([math.exp(-2.0), 1.0, math.exp(-2.0)], dtype=D).tolist()
    sums, total = [torch.zeros_like(f) for f in fields], 0.0
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            w = taps[dx + 1] * taps[dy + 1]
            use = _shift(inner & open_, dx, dy)
            total += w
            for s, f in zip(sums, fields):
                s += w * torch.where(use, _shift(f, dx, dy), f)
    return [s / total for s in sums]


def _backtrace(vx, vy, blocked):
    """Where the air of each cell came from: 0.7 velocity back, walked cell by
    cell and stopped at the first blocked cell."""
    Y, X = vx.shape
    xs = torch.arange(X, device="cuda", dtype=D).expand(Y, X)
    ys = torch.arange(Y, device="cuda", dtype=D)[:, None].expand(Y, X)
    tx, ty = xs - 0.7 * vx, ys - 0.7 * vy
    far = (((0.7 * vx).abs() > 1) | ((0.7 * vy).abs() > 1)) & (tx >= 2) & (tx < X - 2) & (ty >= 2) & (ty < Y - 2)
    at = far.nonzero(as_tuple=True)
    if at[0].numel() == 0:
        return tx, ty
    dx, dy, cx, cy = vx[at], vy[at], xs[at].clone(), ys[at].clone()
    along = dx.abs() > dy.abs()
    big = torch.where(along, dx.abs(), dy.abs())
    sx = torch.where(along, torch.where(dx < 0, 1.0, -1.0), -dx / big)
    sy = torch.where(along, -dy / big, torch.where(dy < 0, 1.0, -1.0))
    limit = (0.7 * big).floor()
    go, hit = limit > 0, torch.zeros_like(along)
    for step in range(int(limit.max().item())):
        nx, ny = cx + sx, cy + sy
        ix, iy = (nx + 0.5).trunc().long(), (ny + 0.5).trunc().long()
        ok = (ix >= 0) & (iy >= 0) & (ix < X) & (iy < Y)
        stop = ~ok | blocked[iy.clamp(0, Y - 1), ix.clamp(0, X - 1)]
        hit |= go & stop
        go &= ~stop
        cx, cy = torch.where(go, nx, cx), torch.where(go, ny, cy)
        go &= step + 1 < limit
    tx[at], ty[at] = torch.where(hit, cx, tx[at]), torch.where(hit, cy, ty[at])
    return tx, ty


def _bilinear(tx, ty, lo, X, Y, hi):
    """Where (tx, ty) lies in the window, and the blend of f(j, i) there."""
    i, j = tx.trunc().long(), ty.trunc().long()
    fx, fy = tx - i, ty - j
    ok = (i >= lo) & (i < X - hi) & (j >= lo) & (j < Y - hi) & (fx >= 0) & (fy >= 0)
    i, j = i.clamp(0, X - 2), j.clamp(0, Y - 2)
    return ok, lambda f: (f(j, i) * (1 - fx) * (1 - fy) + f(j, i + 1) * fx * (1 - fy) +
                          f(j + 1, i) * (1 - fx) * fy + f(j + 1, i + 1) * fx * fy)


def _air_exact(inst):
    X, Y, c = inst.xcells, inst.ycells, inst.config

    def dev(a, dt=D):
        return torch.from_numpy(a.astype(np.float64 if dt == D else np.int64)).to("cuda").reshape(Y, X).to(dt)

    pv, vx, vy, hv, fvx, fvy = (dev(a) for a in (inst.pv, inst.vx, inst.vy, inst.hv, inst.fan_vx, inst.fan_vy))
    blk, hblk, wall = dev(inst.bair, torch.int64) != 0, (dev(inst.bairh, torch.int64) & 8) != 0, dev(inst.wall, torch.int64)
    x = torch.arange(X, device="cuda").expand(Y, X)
    y = torch.arange(Y, device="cuda")[:, None].expand(Y, X)
    rim = (x < 2) | (y < 2) | (x + 2 >= X) | (y + 2 >= Y)
    inner = (x >= 1) & (y >= 1) & (x + 1 < X) & (y + 1 < Y)
    deep = (x > 1) & (y > 1) & (x + 2 < X) & (y + 2 < Y)
    # pressure and velocity
    ex, ey = (torch.where(rim, e + 0.9 * (v - e), v) for v, e in ((vx, c.edge_vx), (vy, c.edge_vy)))
    clear_x = (y >= 1) & (y + 1 < Y) & (((x >= 1) & (x + 1 < X) & blk) | ((x >= 2) & _shift(blk, -1, 0)) |
                                        ((x + 2 < X) & _shift(blk, 1, 0)))
    clear_y = (x >= 1) & (x + 1 < X) & (((y >= 1) & (y + 1 < Y) & blk) | ((y >= 2) & _shift(blk, 0, -1)) |
                                        ((y + 2 < Y) & _shift(blk, 0, 1)))
    ex, ey = ex.masked_fill(clear_x, 0), ey.masked_fill(clear_y, 0)
    e = c.edge_pressure
    cur = torch.where(rim, e + 0.8 * (pv - e), pv)
    div = _shift(ex, -1, 0) - _shift(ex, 1, 0) + _shift(ey, 0, -1) - _shift(ey, 0, 1)
    pv = torch.where(inner, e + 0.9999 * (cur - e) + 0.15 * div, cur)
    nx = c.edge_vx + 0.999 * (ex - c.edge_vx) + 0.2 * (_shift(pv, -1, 0) - _shift(pv, 1, 0))
    ny = c.edge_vy + 0.999 * (ey - c.edge_vy) + 0.2 * (_shift(pv, 0, -1) - _shift(pv, 0, 1))
    nx = nx.masked_fill(blk | _shift(blk, -1, 0) | _shift(blk, 1, 0), 0)
    ny = ny.masked_fill(blk | _shift(blk, 0, -1) | _shift(blk, 0, 1), 0)
    ox, oy = torch.where(inner, nx, ex), torch.where(inner, ny, ey)
    # smoothing, advection, vorticity confinement, fans
    nx, ny, np_ = _smooth([ox, oy, pv], ~blk, inner)
    tx, ty = _backtrace(nx, ny, blk)
    ok, blend = _bilinear(tx, ty, 2, X, Y, 3)
    ok &= ~blk
    nx = torch.where(ok, 0.7 * nx + 0.3 * blend(lambda j, i: ox[j, i]), nx)
    ny = torch.where(ok, 0.7 * ny + 0.3 * blend(lambda j, i: oy[j, i]), ny)
    if c.vorticity_coeff > 0:
        ddx = (_shift(oy, 1, 0) - _shift(oy, -1, 0)).masked_fill(blk | _shift(blk, 1, 0) | _shift(blk, -1, 0), 0)
        ddy = (_shift(ox, 0, 1) - _shift(ox, 0, -1)).masked_fill(blk | _shift(blk, 0, 1) | _shift(blk, 0, -1), 0)
        w = (0.5 * (ddx - ddy)).masked_fill(~deep, 0)
        gx = 0.5 * (_shift(w, 1, 0).abs() - _shift(w, -1, 0).abs())
        gy = 0.5 * (_shift(w, 0, 1).abs() - _shift(w, 0, -1).abs())
        k = c.vorticity_coeff / 5 / (torch.sqrt(gx * gx + gy * gy) + 0.001) * w
        nx, ny = torch.where(deep, nx + k * gy, nx), torch.where(deep, ny - k * gx, ny)
    fan = wall == W.WL_FAN
    nx, ny = torch.where(fan, nx + fvx, nx).clamp(-256, 256), torch.where(fan, ny + fvy, ny).clamp(-256, 256)
    pv = np_.clamp(-256, 256)
    if not c.aheat_enable:
        return {"pv": pv.reshape(-1), "vx": nx.reshape(-1), "vy": ny.reshape(-1), "hv": hv.reshape(-1)}
    # ambient heat and convection
    dh, sx, sy = _smooth([hv, nx, ny], ~hblk, inner)
    tx, ty = _backtrace(sx, sy, hblk)
    ok, blend = _bilinear(tx, ty, 0, X, Y, 1)
    dh = torch.where(ok & ~hblk, 0.7 * dh + 0.3 * blend(lambda j, i: torch.where(hblk[j, i], dh, hv[j, i])), dh)
    dh = torch.where(hblk, hv, dh).clamp(0, 9999).masked_fill(rim, c.ambient_air_temp)
    if c.gravity_mode == 2:
        rx, ry = 0.5 * X - (x + 0.5), 0.5 * Y - (y + 0.5)
        r = torch.sqrt(rx * rx + ry * ry)
        upx, upy = torch.where(r > 0, -rx / r, 0.0), torch.where(r > 0, -ry / r, 0.0)
    else:
        upx, upy = torch.zeros_like(nx), torch.full_like(nx, -1.0)
    if c.convection_mode == 1:
        lift = ((hv - _shift(hv, -1, 0)) * upx + (hv - _shift(hv, 0, -1)) * upy) / 5000
        lift = lift.masked_fill((lift <= 0) | _shift(hblk, 0, -1), 0)
    else:
        lift = ((hv - c.ambient_air_temp) / 10000).clamp(max=0.01)
    vx = torch.where(deep, (nx + lift * upx).clamp(-256, 256), nx)
    vy = torch.where(deep, (ny + lift * upy).clamp(-256, 256), ny)
    return {"pv": pv.reshape(-1), "vx": vx.reshape(-1), "vy": vy.reshape(-1), "hv": dh.reshape(-1)}


def _hot_air(pv, pmap, props, X, Y):
    """Particles that heat the air, in pixel order."""
    pv = pv.reshape(Y, X)
    hot = props.reshape(-1, 32)[:, 11].contiguous().view(torch.float32).to(D)
    ty = (pmap.long() & 0x1FF).reshape(Y, 4, X, 4)
    for dy in range(4):
        for dx in range(4):
            t = ty[:, dy, :, dx]
            h = 4 * hot[t]
            h = torch.where((t == 10) | (t == 97), torch.where(pv < 3.5, h * (3.5 - pv), 0.0), h)
            pv = torch.where(t > 0, pv + h, pv)
    return pv.reshape(-1)


def _gravity_exact(mass, mask, X, Y):
    """-M_GRAV * sum mass (p - m) / |p - m|^3 as a float64 convolution."""
    a, b = 2 * X, 2 * Y
    m = torch.where(mask, mass, 0.0).reshape(Y, X).to(D)
    dx = torch.arange(a, device="cuda", dtype=D)
    dy = torch.arange(b, device="cuda", dtype=D)[:, None]
    dx, dy = torch.where(dx >= X, dx - a, dx), torch.where(dy >= Y, dy - b, dy)
    r2 = dx * dx + dy * dy
    k = torch.where(r2 > 0, -M_GRAV / r2.clamp(min=1) ** 1.5, 0.0)
    f = torch.fft.rfft2(m, s=(b, a))
    out = [torch.fft.irfft2(f * torch.fft.rfft2(k * d), s=(b, a))[:Y, :X] for d in (dx, dy)]
    return [torch.where(mask.reshape(Y, X), o, 0.0).reshape(-1) for o in out]


def _gravtick_exact(case, seed):
    parts, lut, st = _tick_inputs(case, seed)
    X, Y = case["x"], case["y"]
    tool = st["tool_mass"].to(D) * 65536
    tool = torch.where(tool >= 0, tool + 0.5, tool - 0.5).trunc()
    mass = torch.where(st["tool_mass"] != 0, tool, st["mass_prev"].to(D)) / 65536
    gx, gy = _gravity_exact(mass, st["grav_mask"] != 0, X, Y)
    ty, flags = parts["ty"].long(), parts["flags"].long()
    xi, yi = (parts["x"] + 0.5).trunc().long(), (parts["y"] + 0.5).trunc().long()
    ok = (ty > 0) & ((flags & 0x10) == 0) & (xi >= 4) & (yi >= 4) & (xi < 4 * X - 4) & (yi < 4 * Y - 4)
    cell = (yi // 4).clamp(0, Y - 1) * X + (xi // 4).clamp(0, X - 1)
    ok &= ~((st["wall_bmap"][cell] == W.WL_STASIS) & ((st["wall_emap"][cell] & 0xFF) < 8))
    rec = lut.reshape(-1, 12)
    loss = rec[:, 7].contiguous().view(torch.float32).to(D)[ty]
    loss = torch.where((ty == W.PT_SPNG) & ((flags & 8) != 0), 1.0, loss)
    free = (rec[:, 0][ty] & 4) == 0
    out = {"gx": gx, "gy": gy, "mass": None, "mass_prev": None, "tool": None}
    for k, f in (("vx", gx), ("vy", gy)):
        v = parts[k].to(D)
        out[k] = torch.where(ok, v * loss + torch.where(free, f[cell], 0.0), v)
    return out


def _neighbours(a):
    """The six neighbours of every cell of an (y, z, x) grid, zero outside."""
    p = torch.nn.functional.pad(a, (1, 1, 1, 1, 1, 1))
    return (p[1:-1, 1:-1, :-2], p[1:-1, 1:-1, 2:], p[1:-1, :-2, 1:-1], p[1:-1, 2:, 1:-1], p[:-2, 1:-1, 1:-1],
            p[2:, 1:-1, 1:-1])


def _voxel_exact(b, a, iterations):
    n = 64
    g3 = lambda t: t.to(D).reshape(n, n, n)  # noqa: E731
    vx, vy, vz, temp, solid = (g3(t) for t in (a.vx, a.vy, a.vz, a.t, a.solid))
    # listed bricks: occupied share and mean temperature of their cells
    words = b.voxel_a.long() & 0xFFFFFFFF
    full = ((words & 0xFF) != 0).reshape(n, 4, n, 4, n, 4)
    count = full.sum((1, 3, 5)).to(D)
    heat = (((words >> 8) & 0xFFFF).to(D) * 0.125).reshape(n, 4, n, 4, n, 4).masked_fill(~full, 0).sum((1, 3, 5))
    listed_ = torch.zeros(W.VOX_BRICKS, dtype=torch.bool, device="cuda")
    listed_[b.sim_list[:int(b.sim_count[0])].long()] = True
    at = listed_.reshape(32, 32, 32).repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)
    solid = torch.where(at, count / 64, solid)
    temp = torch.where(at, torch.where(count > 0, heat / count.clamp(min=1), 293.15), temp)
    wall = solid > 0.5
    edge = torch.ones(n, n, n, dtype=torch.bool, device="cuda")
    edge[1:-1, 1:-1, 1:-1] = False
    diff = lambda f, k: _neighbours(f)[2 * k + 1] - _neighbours(f)[2 * k]  # noqa: E731
    div = 0.5 * (diff(vx, 0) + diff(vz, 1) + diff(vy, 2))
    p, q = g3(a.p), g3(a.p_tmp)
    for _ in range(iterations):
        p, q = ((sum(_neighbours(p)) - div) / 6).masked_fill(edge | wall, 0), p
    ones = sum(_neighbours(torch.ones_like(vx))) + 1
    mean = lambda f: (f + sum(_neighbours(f))) / ones  # noqa: E731
    clampx = lambda f, k: [torch.where(e, f, m) for e, m in zip(ends[k], _neighbours(f)[2 * k:2 * k + 2])]  # noqa: E731
    idx = torch.arange(n, device="cuda")
    axis = [idx[None, None, :].expand(n, n, n), idx[None, :, None].expand(n, n, n), idx[:, None, None].expand(n, n, n)]
    ends = [(t == 0, t == n - 1) for t in axis]
    out = []
    for f, k, rise in ((vx, 0, 0.0), (vy, 2, 0.02 * (mean(temp) - 293.15)), (vz, 1, 0.0)):
        lo, hi = clampx(p, k)
        v = (f + rise - 0.5 * (hi - lo)) * 0.99
        v = v * 0.9 + mean(f) * 0.1
        lo, hi = clampx(f, k)
        v = v * 0.75 + 0.25 * torch.where(f > 0, lo, torch.where(f < 0, hi, f))
        out.append(v.clamp(-8, 8).masked_fill(wall, 0).reshape(-1))
    u = g3(b.grav_potential)
    rho = g3(b.grav_mass) / 1024
    for _ in range(V.GRAVITY_ITERATIONS):
        u = ((sum(_neighbours(u)) - 8.385539 * rho) / 6).masked_fill(edge, 0)
    force = [(-0.5 * diff(u, k)).masked_fill(edge, 0).reshape(-1) for k in (0, 2, 1)]
    # after an odd number of sweeps the newest pressure is in p_tmp
    p, q = (q, p) if iterations % 2 else (p, q)
    return {"vx": out[0], "vy": out[1], "vz": out[2], "p": p.reshape(-1), "p_tmp": q.reshape(-1), "t": temp.reshape(-1),
            "solid": solid.reshape(-1), "grav_potential": u.reshape(-1), "grav_force_x": force[0],
            "grav_force_y": force[1], "grav_force_z": force[2]}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("air", "frame"):
        g = _gen(seed)
        inst = _instance(g, case["x"], case["y"], case["options"])
        out = {"block_air": None, "block_airh": None, "emap": None}
        out |= _air_exact(inst)
        if kind == "air":
            return out
        out["pv"] = _hot_air(out["pv"], *_particle_map(g, case["x"], case["y"]), case["x"], case["y"])
        mass = torch.from_numpy(inst.mass_fx).to("cuda").to(D) / 65536
        mask = torch.from_numpy(inst.gmask.astype(np.int64)).to("cuda") != 0
        out["gx"], out["gy"] = _gravity_exact(mass, mask, case["x"], case["y"])
        return out
    if kind == "gravity":
        mass, mask = _gravity_inputs(case, seed)
        mass = mass.to(D) / (1.0 if case["f32_mass"] else 65536.0)
        gx, gy = _gravity_exact(mass, mask, case["x"], case["y"])
        return {"gx": gx, "gy": gy}
    if kind == "gravtick":
        return _gravtick_exact(case, seed)
    if kind == "batch":
        # Many ticks of the air have no value in 64 bits: which cells a walk
        # visits and stops at hangs on the last bit of the tick before.
        out = {"pv": None, "vx": None, "vy": None, "hv": None}
        got = []
        for inst in _instances(case, seed):
            mass = torch.from_numpy(inst.mass_fx).to("cuda").to(D) / 65536
            mask = torch.from_numpy(inst.gmask.astype(np.int64)).to("cuda") != 0
            got.append([f.cpu() for f in _gravity_exact(mass, mask, inst.xcells, inst.ycells)])
        out["gx"], out["gy"] = torch.cat([a for a, _ in got]), torch.cat([b for _, b in got])
        return out
    got = [_voxel_exact(b, a, case["iterations"]) for b, a in _worlds(case, seed)[0]]
    return {"pv": None, "grav_mass": None} | {k: torch.stack([d[k] for d in got]) for k in got[0]}
