"""The engine's performance cases: what its users run, as plain descriptions with a way to make
each one's inputs, run one pass of it and say what the pass cannot do without.

A pass starts from a scene's particles in host memory (`FluidSim.reset`), advances the scene
frame by frame (a frame is 4 substeps of 1/240 s) and reads the particles and the pressure back,
as a headless run of a scene does; the solve cases hand the library a linear system that lives
on the device; the scene case turns shapes into the solid fields.

Kinds:
  solve   `pressure_solve_static` on a device-resident two-column system (an embedding host
          that owns the device memory).
  dam     a water dam break: one liquid, explicit viscosity, one pressure solve per substep.
  honey   a dam break of the built-in honey: implicit viscosity, two pressure solves.
  layers  built-in honey, water and olive oil stacked: concentration families, an immiscible
          group, implicit viscosity.
  pour    the full-physics pour: eight liquids, heater, heat, surface tension, implicit
          viscosity, plain FP32 or mixed-precision pressure solves.
  batch   many uneven tanks advanced together (`Batch.step`).
  serve   changing subsets of resident tanks advanced launch by launch (`Batch.step_subset`).
  frame   a rendered run: substeps, the render side's cell passes and the particle fields of a
          view, images read back at the end.
  scene   `Scene.rasterize` on the device.
"""
import math

import numpy as np
import torch

import sprout_gb300 as S
from sprout_gb300 import workloads as WL

FRAME = 4              # substeps of a 1/60 s frame at the configurations' fixed 240 Hz
DT = 1.0 / 240.0
STATIC_CELLS = 512 * 288   # the largest grid the allocation-free solve takes


def listed():
    return [
        # the smallest call: one solve of the smallest benchmark grid, launch and barrier latency
        {"name": "solve_128x72", "kind": "solve", "w": 128, "h": 72, "tol": 1e-5},
        # the largest grid the allocation-free solve takes, ragged against the 16 x 16 tiles
        {"name": "solve_509x287", "kind": "solve", "w": 509, "h": 287, "tol": 1e-5},
        # the smallest tank of the batched and serving mixes, stepped alone (interactive use)
        {"name": "dam_128x72", "kind": "dam", "w": 128, "h": 72, "frames": 16},
        # the first benchmark configuration: a water dam break on 384 x 216
        {"name": "dam_384x216", "kind": "dam", "w": 384, "h": 216, "frames": 12},
        # the largest published scene of the reference: a dam break of 1.04 M water particles
        {"name": "dam_1600x900", "kind": "dam", "w": 1600, "h": 900, "frames": 12},
        # the second configuration: honey, water and olive oil on 512 x 288
        {"name": "layers_512x288", "kind": "layers", "w": 512, "h": 288, "frames": 10},
        # the third configuration, the benchmark's default: the full-physics pour on 1024 x 576
        {"name": "pour_1024x576", "kind": "pour", "w": 1024, "h": 576, "frames": 12, "precision": "plain"},
        # the same liquids with mixed-precision solves on an odd, ragged grid
        {"name": "pour_mixed_701x397", "kind": "pour", "w": 701, "h": 397, "frames": 12, "precision": "mixed"},
        # the batched configuration's mix (uneven dam breaks of one or two liquids), 20 tanks
        {"name": "batch_20", "kind": "batch", "tanks": 20, "w": 1024, "frames": 5, "precision": "plain"},
        # the serving mix: 16 of 20 resident small tanks per launch, another 16 each time
        {"name": "serve_20", "kind": "serve", "tanks": 20, "w": 384, "launches": 24, "subset": 16, "precision": "mixed"},
        # a rendered run: cell optics, light, flow map and the particle fields of a 1080p view
        {"name": "frame_512x288", "kind": "frame", "w": 512, "h": 288, "frames": 8, "view_w": 1920, "view_h": 1080},
        # a scene with a dozen solids turned into the tank's solid fields
        {"name": "scene_1024x576", "kind": "scene", "w": 1024, "h": 576, "shapes": 12},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _size(rng, lo, hi):
    """A grid of about 16:9, its width spread over [lo, hi] by its logarithm, any remainder."""
    w = int(round(_log(rng, lo, hi)))
    h = int(round(w * rng.uniform(0.45, 0.7)))
    return max(w, 48), max(h, 32)


def draw(rng):
    kind = rng.choice(["solve", "solve", "dam", "dam", "dam", "honey", "layers", "layers", "pour", "pour", "batch", "serve",
                       "frame", "scene"])
    if kind == "solve":
        w, h = _size(rng, 64, 512)
        return {"kind": kind, "w": w, "h": min(h, STATIC_CELLS // w), "tol": rng.choice([1e-4, 1e-5])}
    if kind in ("dam", "honey", "layers"):
        w, h = _size(rng, 96, 1024 if kind == "dam" else 640)
        return {"kind": kind, "w": w, "h": h, "frames": rng.randint(4, 10)}
    if kind == "pour":
        w, h = _size(rng, 128, 1000)
        return {"kind": kind, "w": w, "h": h, "frames": rng.randint(4, 10), "precision": rng.choice(["plain", "mixed"])}
    if kind == "batch":
        return {"kind": kind, "tanks": rng.randint(3, 16), "w": rng.choice([256, 512, 1024]), "frames": rng.randint(2, 5),
                "precision": rng.choice(["plain", "mixed"])}
    if kind == "serve":
        n = rng.randint(6, 20)
        return {"kind": kind, "tanks": n, "w": rng.choice([256, 384]), "launches": rng.randint(8, 24),
                "subset": rng.randint(2, n), "precision": rng.choice(["plain", "mixed"])}
    if kind == "frame":
        w, h = _size(rng, 128, 640)
        vw = int(round(_log(rng, 480, 1920)))
        return {"kind": kind, "w": w, "h": h, "frames": rng.randint(3, 8), "view_w": vw, "view_h": int(round(vw * 0.5625))}
    w, h = _size(rng, 96, 1024)
    return {"kind": "scene", "w": w, "h": h, "shapes": rng.randint(1, 16)}


# ---- inputs ---------------------------------------------------------------------------------

def _stir(tank, seed):
    """The tank with its liquid set moving by the seed: a few divergence-free eddies of up to
    0.2 m/s that vanish at the walls."""
    rng = np.random.default_rng(seed)
    w, h = float(tank.w), float(tank.h)
    modes = [(i, j, float(rng.uniform(-1.0, 1.0))) for i in (1, 2) for j in (1, 2, 3)]
    speed = 0.2 / tank.settings["cell_size"] / 6.0   # cells/s a mode

    def stir(parts):
        x, y = parts["pos"][:, 0].astype(np.float64) / w, parts["pos"][:, 1].astype(np.float64) / h
        vx, vy = np.zeros(len(parts)), np.zeros(len(parts))
        for i, j, a in modes:   # of the stream function a sin(i pi x / w) sin(j pi y / h)
            k = a * speed / math.hypot(i / w, j / h)
            vx += k * j / h * np.sin(i * math.pi * x) * np.cos(j * math.pi * y)
            vy -= k * i / w * np.cos(i * math.pi * x) * np.sin(j * math.pi * y)
        parts["vel"][:, 0] = vx
        parts["vel"][:, 1] = vy
        return parts
    tank.prepare = stir
    return tank


def _tanks(case, seed):
    kind, w = case["kind"], case["w"]
    if kind in ("batch", "serve"):
        # sizes up to the case's width, from the mix's own list and weights; the liquids and
        # blocks of tank k are the mix's k-th draw
        n_sizes = sum(1 for s in WL.UNEVEN_SIZES if s[0] <= w)
        wt = np.array(WL.SERVING_WEIGHTS if kind == "serve" else [1.0] * 6)
        wt[n_sizes:] = 0.0
        return [_stir(t, seed * 64 + k) for k, t in
                enumerate(WL.uneven_dam_breaks(case["tanks"], seed=7, weights=list(wt / wt.sum())))]
    h = case["h"]
    if kind == "dam":
        t = WL.dam_break(w, h, cell=0.768 / w, width=0.4, height=0.6, tol=1e-5)
        if w == 1600:   # the reference's own scene: 1.04 M particles
            t.fills = [([0.0, 0.0, 0.3 * w, 0.6 * h], 0, None)]
    elif kind == "honey":
        t = WL.dam_break(w, h, cell=0.768 / w, width=0.4, height=0.6, tol=1e-5, mat=1, extra={"viscosity_tol": 1e-5})
    elif kind == "layers":
        t = WL.stratified(w, h, cell=1.024 / w, tol=1e-5, builtins=True)
    elif kind == "frame":
        t = WL.dam_break(w, h, cell=0.768 / w, width=0.4, height=0.6, tol=1e-4)
    else:
        t = WL.full_physics(w, h, cell=1.024 / w, n_liquids=8, seed=0, heater_rows=8, tol=1e-5)
    return [_stir(t, seed)]


def _system(case, seed):
    """A two-column pressure system on the device: a liquid body with a wavy surface under air
    (Dirichlet there, nothing through the walls), layered densities, right-hand sides of a
    divergence (column 0) and a density error (column 1)."""
    w, h = case["w"], case["h"]
    g = torch.Generator(device="cpu").manual_seed(int(seed))
    u = torch.rand(8, generator=g, dtype=torch.float64)
    x = torch.arange(w, dtype=torch.float64)[None, :] + 0.5
    y = torch.arange(h, dtype=torch.float64)[:, None] + 0.5
    surface = h * (0.6 + 0.08 * torch.sin(2 * math.pi * (x / w * 1.5 + u[0])) + 0.05 * torch.sin(2 * math.pi * (x / w * 5 + u[1])))
    open_ = ((x > 2) & (x < w - 2) & (y > 2) & (y < h - 2)).expand(h, w)
    liquid = open_ & (y < surface)
    rho = (1.0 + 9.0 * (torch.sin(2 * math.pi * (y / h * 2 + x / w * 0.5 + u[2])) > 0)).expand(h, w)
    A = torch.zeros(h, w, 4, dtype=torch.float64)
    for q, (dx, dy) in enumerate([(-1, 0), (1, 0), (0, -1), (0, 1)]):
        nr = torch.roll(rho, (-dy, -dx), (0, 1))
        no = torch.roll(open_, (-dy, -dx), (0, 1))
        nl = torch.roll(liquid, (-dy, -dx), (0, 1))
        c = torch.where(nl, 2.0 / (rho + nr), 1.0 / rho)
        A[:, :, q] = torch.where(liquid & no, c, torch.zeros(()).double())
    A = A.float()
    D = torch.where(liquid, A.sum(2), torch.zeros(()))
    wave = lambda k, p: torch.sin(2 * math.pi * (x / w * k + p)) * torch.cos(2 * math.pi * (y / h * k * 0.6 + p))
    div = 0.02 * wave(2, u[3]) + 0.01 * wave(9, u[4]) + 0.005 * torch.randn(h, w, generator=g, dtype=torch.float64)
    err = 0.002 * torch.randn(h, w, generator=g, dtype=torch.float64) + 0.001 * wave(3, u[5])
    B = torch.stack([div, err], 2).float() * liquid[:, :, None]
    return A.reshape(-1, 4).contiguous(), D.reshape(-1).contiguous(), B.reshape(-1, 2).contiguous()


def _scene(case, seed):
    rng = np.random.default_rng(seed)
    w, h = case["w"], case["h"]
    sc = S.Scene(w, h)
    for k in range(case["shapes"]):
        c = (float(rng.uniform(0.1, 0.9) * w), float(rng.uniform(0.1, 0.9) * h))
        temp = float(rng.uniform(20.0, 200.0)) if k % 4 == 3 else None
        if k % 2:
            sc.add_circle(c, float(rng.uniform(0.02, 0.1) * h), temp)
        else:
            sc.add_box(c, (float(rng.uniform(0.02, 0.12) * w), float(rng.uniform(0.01, 0.06) * h)),
                       float(rng.uniform(-1.5, 1.5)), temp)
    return sc


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        A, D, B = (t.cuda() for t in _system(case, seed))
        return {"case": case, "A": A, "D": D, "B": B, "x0": torch.zeros_like(B)}
    if kind == "scene":
        return {"case": case, "scene": _scene(case, seed)}
    built = [t.engine() for t in _tanks(case, seed)]
    st = {"case": case, "sims": [b[0] for b in built], "parts": [b[1] for b in built]}
    if kind in ("batch", "serve"):
        st["batch"] = S.Batch(st["sims"], case["precision"])
    elif case.get("precision") == "mixed":
        st["sims"][0].set_precision("mixed")
    return st


# ---- one pass -------------------------------------------------------------------------------

def _particles(sim):
    """The particles as they come: motion (position, velocity, affine matrix, concentration),
    tags (kind, id) and temperature, as views of the downloaded records."""
    p = sim.download_particles()
    f = p.view(np.float32).reshape(-1, 12)
    return {"motion": f[:, :9], "tags": p.view(np.int32).reshape(-1, 12)[:, 9:11], "heat": f[:, 11]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        x = state["x0"].clone()
        iters, res = S.pressure_solve_static(case["w"], case["h"], state["A"].data_ptr(), state["D"].data_ptr(),
                                             state["B"].data_ptr(), x.data_ptr(), case["tol"], 1e-2, 60)
        return {"x": x, "iters": np.array(iters, np.int32), "residual": res}
    if kind == "scene":
        sdf, solid, region, temp = state["scene"].rasterize(device=True)
        return {"sdf": sdf, "solid": solid, "region": region.view(np.int32), "temp": temp}
    for sim, parts in zip(state["sims"], state["parts"]):
        sim.reset(parts)
    if kind == "batch":
        for _ in range(case["frames"]):
            state["batch"].step(FRAME)
        return [_particles(sim) for sim in state["sims"]]
    if kind == "serve":
        n, m = case["tanks"], case["subset"]
        for k in range(case["launches"]):
            state["batch"].step_subset([(k * 5 + j) % n for j in range(m)])
        return [_particles(sim) for sim in state["sims"]]
    sim = state["sims"][0]
    if kind == "frame":
        w, h, vw, vh = case["w"], case["h"], case["view_w"], case["view_h"]
        for _ in range(case["frames"]):
            sim.step(FRAME, FRAME * DT)
            sim.render(1.0 / 60.0)
            sim.draw((w / 2.0, h / 2.0), vw / w, (vw, vh))
        return {"sharp": sim.download_draw("sharp"), "wide": sim.download_draw("wide"),
                "layers": sim.download_render("smoothed"), "glow": sim.download_render("glow")}
    for _ in range(case["frames"]):
        sim.step(FRAME, FRAME * DT)
    return {**_particles(sim), "pressure": sim.download_pressure()}


# ---- what a pass cannot do without ----------------------------------------------------------

def work(case):
    """Bytes: per substep each particle (48 B) read and written once and each cell's carried
    state (solids 16 B, pressure 8 B) read and its pressure written, the host copies of a pass
    (particles in and out, images out) once. FLOP: per particle 200 (a nine-point gather and
    scatter with the affine matrix), per cell and substep 12 conjugate-gradient iterations of
    the two-column five-point operator with its V-cycle (about 4/3 x 120). A solve case reads
    its system and writes its solution once."""
    kind = case["kind"]
    if kind == "solve":
        n = case["w"] * case["h"]
        return {"bytes": n * (16 + 4 + 8 + 8 + 8), "flops": n * 12 * 160}
    if kind == "scene":
        n = case["w"] * case["h"]
        return {"bytes": n * 28, "flops": n * 20 * case["shapes"]}
    share = {"dam": 0.24, "honey": 0.24, "layers": 0.6, "pour": 0.97, "frame": 0.24}
    if kind in ("batch", "serve"):
        cells = [t.w * t.h for t in _tanks(case, 0)]
        steps = FRAME * case["frames"] if kind == "batch" else case["launches"] * case["subset"] / case["tanks"]
        n, parts = sum(cells), 4 * 0.22 * sum(cells)
    else:
        n = case["w"] * case["h"]
        parts = 4 * share[kind] * n
        steps = FRAME * case["frames"]
    out = 96 * parts + 8 * n
    if kind == "frame":
        out = 48 * parts + 16 * case["view_w"] * case["view_h"] + 200 * n
    return {"bytes": steps * (96 * parts + 32 * n) + out, "flops": steps * (200 * parts + 12 * 160 * n)}


def exact(case, seed):
    """The solve cases' solution in 64 bits (conjugate gradients with the diagonal to 1e-12).
    The other cases advance a tank by a chain of single-precision substeps or draw images of
    one: they have no closed form to compare with."""
    if case["kind"] != "solve":
        return None
    w, h = case["w"], case["h"]
    A, D, B = (t.cuda().double() for t in _system(case, seed))
    A, D, B = A.reshape(h, w, 4), D.reshape(h, w, 1), B.reshape(h, w, 2)
    on = D > 0
    inv = torch.where(on, 1.0 / torch.where(on, D, torch.ones_like(D)), torch.zeros_like(D))
    wt = [A[:, :, q:q + 1] * on * torch.roll(on, s, d) for q, (s, d) in enumerate([(1, 1), (-1, 1), (1, 0), (-1, 0)])]

    def apply(p):
        q = D * p
        for c, (s, d) in zip(wt, [(1, 1), (-1, 1), (1, 0), (-1, 0)]):
            q = q - c * torch.roll(p, s, d)
        return q
    x = torch.zeros_like(B)
    r = B.clone()
    z = inv * r
    p = z.clone()
    rz = (r * z).sum((0, 1))
    b2 = (B * B).sum((0, 1)).clamp_min(1e-300)
    for it in range(20000):
        q = apply(p)
        a = rz / (p * q).sum((0, 1)).clamp_min(1e-300)
        x = x + a * p
        r = r - a * q
        z = inv * r
        new = (r * z).sum((0, 1))
        p = z + (new / rz.clamp_min(1e-300)) * p
        rz = new
        if it % 50 == 49 and float(((r * r).sum((0, 1)) / b2).max()) < 1e-24:
            break
    return {"x": x.reshape(-1, 2), "iters": None, "residual": None}
