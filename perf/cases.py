"""The work that programs have this framework do, as cases that can be timed and compared.

Every case goes through the public Python package or the C-ABI, at the sizes that the repository's configurations, tests
and benchmark use and at generic ones beside them (sides that are no power of two, oblong grids, ragged particle
counts).  A pass hands its result to the host the way such a program does: particles through the pipelined Vec2x8 read
into pinned memory, a frame through the frame read, sorted keys as device tensors.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "apic-fluid-simulation_gb300"))
import apic_gb300 as A  # noqa: E402

GRAVITY, DAMPING, CFL = -9.81, 0.1, 5.0
SOLVERS = {"reference": A.SOLVER_REFERENCE, "fp32": A.SOLVER_REL_FP32, "mixed": A.SOLVER_REL_MIXED}


def listed():
    return [
        # the smallest scene in use: the viewer's loop on a 64 x 64 grid, where launches and latency are all there is
        {"name": "frame_64", "kind": "frames", "scene": "default", "width": 64, "height": 64, "cell": 1 / 64,
         "solver": "reference", "dt": 1 / 60, "drag": False},
        # the viewer as it starts: 256 x 256 cells of 0.075, the user dragging the fluid with the mouse in every frame
        {"name": "frame_256_drag", "kind": "frames", "scene": "default", "width": 256, "height": 256, "cell": 0.075,
         "solver": "reference", "dt": 1 / 60, "drag": True},
        # the reference's own benchmark at its largest: cells of 1.0, nine particles in each, its solver, a run of
        # updates from the same warmed-up state
        {"name": "criterion_1024", "kind": "rollout", "scene": "default", "width": 1024, "height": 1024, "cell": 1.0,
         "solver": "reference", "dt": 0.016, "updates": 10},
        # the plain dam break at 128 x 128, stepped and read back update by update
        {"name": "dam_128", "kind": "frames", "scene": "dam", "width": 128, "height": 128, "cell": 1 / 128,
         "solver": "mixed", "dt": 1 / 240, "drag": False},
        # the large single scene (dam break and a falling disk): four updates from a checkpoint, as a program does that
        # tries something from the same state again and again
        {"name": "rollout_1024", "kind": "rollout", "scene": "disk", "width": 1024, "height": 1024, "cell": 1 / 1024,
         "solver": "mixed", "dt": 1 / 480, "updates": 4},
        # the same at an ordinary size
        {"name": "rollout_256", "kind": "rollout", "scene": "disk", "width": 256, "height": 256, "cell": 1 / 256,
         "solver": "mixed", "dt": 1 / 240, "updates": 8},
        # an oblong grid whose sides are no powers of two and stop halving early, with the plain FP32 solver
        {"name": "noise_1000x600", "kind": "frames", "scene": "noise", "width": 1000, "height": 600, "cell": 1 / 1000,
         "solver": "fp32", "dt": 1 / 1000, "drag": False},
        # the largest: 33 million particles over a noise mask on 4096 x 4096 cells, sorted in every update
        {"name": "stress_4096", "kind": "frames", "scene": "noise", "width": 4096, "height": 4096, "cell": 1 / 4096,
         "solver": "mixed", "dt": 1 / 1000, "drag": False},
        # many independent scenes of uneven size stepped together, in the form that the library picks
        {"name": "batch_24", "kind": "batch", "count": 24, "low": 64, "high": 256, "mix": 3, "dt": 1 / 240},
        # a server's burst: requests for whole scenes come in at once, run side by side, and their results are fetched
        {"name": "serve_12", "kind": "serve", "count": 12, "low": 64, "high": 256, "mix": 4, "steps": 20,
         "dt": 1 / 240},
        # the Morton sort alone, on a caller's own device arrays
        {"name": "sort_1m", "kind": "sort", "n": 1000003, "width": 1024, "height": 1024},
        # the headless particle view of the large scene in a full HD frame
        {"name": "render_1080p", "kind": "render", "side": 1024, "frame_w": 1920, "frame_h": 1080},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _side(rng, low, high):
    """An even side (grids with particles need one): a third of the draws a power of two, the large ones at least a
    multiple of 8, so that the grid halves a few times."""
    s = _log_int(rng, low, high)
    if rng.random() < 0.33:
        s = 1 << int(round(math.log2(s)))
    else:
        m = 2 if s < 128 else 4 if s < 256 else 8
        s = s // m * m
    return max(low, min(high, s))


def draw(rng):
    kind = rng.choice(["frames", "frames", "frames", "rollout", "batch", "serve", "sort", "render"])
    if kind == "frames":
        how = rng.choice(["default", "dam", "noise"])
        if how == "default":
            s, cell = _side(rng, 64, 768), rng.choice(["unit", "gui", "one"])
            return {"kind": kind, "scene": how, "width": s, "height": s,
                    "cell": {"unit": 1 / s, "gui": 0.075, "one": 1.0}[cell], "solver": "reference",
                    "dt": rng.choice([1 / 60, 0.016]), "drag": rng.random() < 0.5}
        w, h = _side(rng, 64, 1536), _side(rng, 64, 1536)
        return {"kind": kind, "scene": how, "width": w, "height": h, "cell": 1 / w,
                "solver": rng.choice(["mixed", "mixed", "fp32"]),
                "dt": 1 / rng.choice([240, 480] if how == "dam" else [500, 1000]), "drag": rng.random() < 0.3}
    if kind == "rollout":
        s = _side(rng, 64, 1024)
        return {"kind": kind, "scene": rng.choice(["dam", "disk"]), "width": s, "height": s, "cell": 1 / s,
                "solver": "mixed", "dt": 1 / rng.choice([240, 480]), "updates": rng.randint(2, 6)}
    if kind in ("batch", "serve"):
        low = rng.choice([64, 96])
        c = {"kind": kind, "count": _log_int(rng, 4, 24), "low": low, "high": rng.choice([160, 256]),
             "mix": rng.randrange(1000), "dt": 1 / 240}
        return {**c, "steps": rng.randint(5, 20)} if kind == "serve" else c
    if kind == "sort":
        return {"kind": kind, "n": _log_int(rng, 1000, 1 << 20), "width": _side(rng, 64, 4096),
                "height": _side(rng, 64, 4096)}
    big = rng.random() < 0.5
    return {"kind": kind, "side": _side(rng, 64, 768), "frame_w": 1920 if big else 1280,
            "frame_h": 1080 if big else 720}


# ---- inputs -----------------------------------------------------------------

def _fluid_cells(case):
    """Mask of the cells that hold fluid (height x width) for a scene on a domain of width 1."""
    w, h = case["width"], case["height"]
    x = (np.arange(w) + 0.5) / w
    y = (np.arange(h) + 0.5) / w
    inner = np.zeros((h, w), bool)
    inner[2:h - 2, 2:w - 2] = True
    if case["scene"] == "noise":
        # value noise, the same for every seed: lattice values of period 1/64 of the width, bilinear between them,
        # fluid above 0.5
        period = 1 / 64 if w >= 512 else 1 / 16
        lat = np.random.default_rng(2).random((int(math.ceil(h / w / period)) + 2, int(math.ceil(1 / period)) + 2)).astype(np.float32)
        fx, fy = x / period, y / period
        ix, iy = fx.astype(int), fy.astype(int)
        tx, ty = (fx - ix).astype(np.float32)[None, :], (fy - iy).astype(np.float32)[:, None]
        low = lat[iy][:, ix] * (1 - tx) + lat[iy][:, ix + 1] * tx
        high = lat[iy + 1][:, ix] * (1 - tx) + lat[iy + 1][:, ix + 1] * tx
        return inner & (low * (1 - ty) + high * ty > 0.5), None
    top = h / w
    if case["scene"] == "dam":
        return inner & ((x < 0.4)[None, :] & (y < 0.6 * top)[:, None]), None
    disk = (x[None, :] - 0.7) ** 2 + (y[:, None] - 0.8 * top) ** 2 < 0.08 ** 2
    return inner & (((x < 0.5)[None, :] & (y < 0.5 * top)[:, None]) | disk), disk


def _particles(case, seed):
    """Four jittered particles in each fluid cell: float32 positions and velocities."""
    rng = np.random.default_rng(seed)
    mask, disk = _fluid_cells(case)
    cy, cx = np.nonzero(mask)
    n = 4 * len(cx)
    sub = np.tile(np.array([[0.0, 0.0], [0.5, 0.0], [0.0, 0.5], [0.5, 0.5]], np.float32), (len(cx), 1))
    dx = np.float32(case["cell"])
    px = (np.repeat(cx, 4).astype(np.float32) + sub[:, 0] + 0.5 * rng.random(n, np.float32)) * dx
    py = (np.repeat(cy, 4).astype(np.float32) + sub[:, 1] + 0.5 * rng.random(n, np.float32)) * dx
    vx, vy = np.zeros(n, np.float32), np.zeros(n, np.float32)
    if case["scene"] == "noise":
        vx = 0.5 * rng.standard_normal(n, np.float32)
        vy = 0.5 * rng.standard_normal(n, np.float32)
    elif disk is not None:
        vy[np.repeat(disk[cy, cx], 4)] = -2.0
    return px, py, vx, vy


def _sides(case):
    rng = random.Random(case["mix"])
    return [_log_int(rng, case["low"] / 8, case["high"] / 8) * 8 for _ in range(case["count"])]


def _props():
    return A.WorldProperties(gravity=GRAVITY, border_damping=DAMPING, cfl=CFL, solve_error=1e-5)


def _sim(case, seed):
    sim = A.Apic.new(case["width"], case["height"], case["cell"], _props())
    if case["scene"] == "default":
        # the block that the constructor fills, moving as a whole
        v = np.zeros(sim.num_chunks * 8, np.float32)
        rng = np.random.default_rng(seed)
        for f in ("vel_x", "vel_y"):
            v[:sim.num_particles] = 0.05 * case["cell"] / case["dt"] * rng.uniform(-1, 1)
            sim.write_field(f, v)
    else:
        sim.set_particles(*_particles(case, seed))
    sim.set_solver(SOLVERS[case["solver"]], 1e-6, 500)
    return sim


def _host(floats):
    return torch.empty(floats, dtype=torch.float32, pin_memory=True)


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "options": A.DebugOptions()}
    if kind in ("frames", "rollout"):
        sim = s["sim"] = _sim(case, seed)
        floats = sim.num_chunks * 16
        s["pos"], s["vel"] = _host(floats), _host(floats)
        if kind == "rollout":
            for _ in range(2):
                sim.update(s["options"], case["dt"])
            blob = np.frombuffer(sim.snapshot(), np.uint8)
            s["checkpoint"] = torch.empty(blob.size, dtype=torch.uint8, pin_memory=True)
            s["checkpoint"].numpy()[:] = blob
        elif case["drag"]:
            span = case["width"] * case["cell"]
            rng = random.Random(seed)
            s["drags"] = [(rng.uniform(0.1, 0.9) * span, rng.uniform(0.05, 0.4) * span, 0.08 * span,
                           rng.choice([-1.0, 1.0]) * span * 5.0) for _ in range(64)]
            s["frame"] = 0
    elif kind == "batch":
        s["sims"] = [_sim({"scene": "dam", "width": n, "height": n, "cell": 1 / n, "solver": "mixed"}, seed * 100 + i)
                     for i, n in enumerate(_sides(case))]
        s["floats"] = [sim.num_chunks * 16 for sim in s["sims"]]
        s["pos"], s["vel"] = _host(sum(s["floats"])), _host(sum(s["floats"]))
    elif kind == "serve":
        s["scenes"] = [A.scene_params(A.SCENE_DAM_BREAK_DISK if i % 2 else A.SCENE_DAM_BREAK, n, cell_size=1 / n,
                                      seed=(seed * 100 + i) % (1 << 31), fluid_x=0.4, fluid_y=0.5,
                                      disk=(0.7, 0.8, 0.08), disk_v=(0.0, -2.0))
                       for i, n in enumerate(_sides(case))]
        s["props"] = _props()
    elif kind == "sort":
        # particles as a step leaves them: in the order of an earlier sort by cell, most of them moved since
        g = torch.Generator(device="cuda").manual_seed(seed)
        n, w, h = case["n"], case["width"], case["height"]
        at = torch.sort(torch.randint(0, w * h, (n,), device="cuda", generator=g)).values
        move = torch.randn(2, n, device="cuda", generator=g)
        dx = 1.0 / w
        s["dx"] = dx
        s["x"] = ((at % w).float() + 0.5 + move[0]) * dx
        s["y"] = (torch.div(at, w, rounding_mode="floor").float() + 0.5 + move[1]) * dx
        s["keys"] = torch.empty(n, dtype=torch.int32, device="cuda")
        s["vals"] = torch.empty(n, dtype=torch.int32, device="cuda")
        s["lib"] = A.load_library()
    elif kind == "render":
        n = case["side"]
        s["sim"] = _sim({"scene": "disk", "width": n, "height": n, "cell": 1 / n, "solver": "mixed"}, seed)
        for _ in range(2):
            s["sim"].update(s["options"], 1 / 480)
        w, h = case["frame_w"], case["frame_h"]
        s["view"] = A.render_params(w, h, scale=float(h), pick=(0.3 * w, 0.7 * h))
    torch.cuda.synchronize()
    return s


# ---- one pass ---------------------------------------------------------------

def _read(sims, floats, pos, vel):
    """Positions and velocities of the scenes into pinned memory, one after another."""
    at = 0
    for sim, n in zip(sims, floats):
        sim.read_vec2x8_async(0, pos.data_ptr() + 4 * at, n)
        sim.read_vec2x8_async(1, vel.data_ptr() + 4 * at, n)
        at += n
    for sim in sims:
        sim.read_wait()
    return [pos, vel]


def _check(code, what):
    if code != A.OK:
        raise RuntimeError("%s: status %d" % (what, code))


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "frames":
        sim = s["sim"]
        if case["drag"]:
            sim.add_radial_force(*s["drags"][s["frame"] % 64])
            s["frame"] += 1
        sim.update(s["options"], case["dt"])
        return _read([sim], [s["pos"].numel()], s["pos"], s["vel"])
    if kind == "rollout":
        sim, blob = s["sim"], s["checkpoint"]
        _check(A.load_library().apic_restore(sim._h, ctypes.c_void_p(blob.data_ptr()), blob.numel()), "apic_restore")
        for _ in range(case["updates"]):
            sim.update(s["options"], case["dt"])
        return _read([sim], [s["pos"].numel()], s["pos"], s["vel"])
    if kind == "batch":
        A.update_batch(s["sims"], s["options"], case["dt"])
        return _read(s["sims"], s["floats"], s["pos"], s["vel"])
    if kind == "serve":
        server = A.Server(16 << 30, 64, keep_results=True)
        ids = [server.submit(scene, s["props"], case["steps"], case["dt"]) for scene in s["scenes"]]
        while server.step().completed or server.stats().completed + server.stats().failed < len(ids):
            pass
        got = [server.result_positions(i) for i in ids]
        server.close()
        return got
    if kind == "sort":
        _check(s["lib"].apic_morton_sort_noalloc(
            s["x"].data_ptr(), s["y"].data_ptr(), case["n"], case["width"], case["height"], s["dx"],
            s["keys"].data_ptr(), s["vals"].data_ptr(), torch.cuda.current_stream().cuda_stream), "sort")
        return [s["keys"], s["vals"]]
    frame, st = s["sim"].render(s["view"])
    return [frame, st.valid, st.nan, st.out_of_bounds, st.picked]


# ---- what a pass cannot do without ------------------------------------------

def _count(case):
    """Particles of a scene, near enough."""
    w, h = case["width"], case["height"]
    if case["scene"] == "default":
        return 9 * (w - 9) * (h // 2 - 5)
    return int(4 * w * h * {"dam": 0.24, "disk": 0.27, "noise": 0.5}[case["scene"]])


def work(case):
    kind = case["kind"]
    # an update reads and writes a particle's nine numbers once; 16 more bytes of each particle go to the host
    if kind == "frames":
        n = _count(case)
        return {"bytes": 88 * n, "flops": 150 * n}
    if kind == "rollout":
        n = _count(case)
        return {"bytes": (36 + 16 + 72 * case["updates"]) * n, "flops": 150 * n * case["updates"]}
    if kind in ("batch", "serve"):
        n = sum(_count({"scene": "dam", "width": s, "height": s}) for s in _sides(case))
        k = case.get("steps", 1)
        return {"bytes": (16 + 72 * k) * n, "flops": 150 * n * k}
    if kind == "sort":
        return {"bytes": 16 * case["n"], "flops": 0}
    n = _count({"scene": "disk", "width": case["side"], "height": case["side"]})
    return {"bytes": 16 * n + 4 * case["frame_w"] * case["frame_h"], "flops": 0}


# ---- 64-bit values ----------------------------------------------------------

def exact(case, seed):
    """The first update of a scene with a relative solver, in 64 bits.

    None where there is no such value: the reference's solver stops at an absolute residual, long before its answer is
    a property of the inputs, and from the second update on a rounding moves single particles over the edges of the
    sort's cells, which renumbers the slots that seed the advection's jitter.  Keys, bytes and counts are whole."""
    if case["kind"] != "frames" or case["solver"] == "reference" or case["drag"]:
        return None
    px, py, vx, vy = _particles(case, seed)
    if float(np.sqrt(vx * vx + vy * vy).max()) * case["dt"] > 0.9 * CFL * case["cell"]:
        return None  # more than one substep
    return _first_update(case, px, py, vx, vy)


def _spread(v):
    for shift, keep in ((8, 0x00FF00FF), (4, 0x0F0F0F0F), (2, 0x33333333), (1, 0x55555555)):
        v = (v | (v << shift)) & keep
    return v


def _shift(a, dy, dx, fill=0):
    """b[y, x] = a[y + dy, x + dx], `fill` outside."""
    b = torch.full_like(a, fill)
    h, w = a.shape
    b[max(0, -dy):h - max(0, dy), max(0, -dx):w - max(0, dx)] = \
        a[max(0, dy):h - max(0, -dy), max(0, dx):w - max(0, -dx)]
    return b


SIDES = ((0, -1), (0, 1), (-1, 0), (1, 0))  # left, right, below, above


def _theta(outside, inside):
    diff = inside - outside
    t = ((inside - 4.5) / diff).clamp(0.1, 1.0)
    return torch.where(diff.abs() <= 1e-5, torch.ones_like(t), t)


def _corners(gx, gy, ox, oy, w, h):
    """The four nodes (clamped into w x h), weights and fractions of a bilinear stencil offset by (ox, oy)."""
    x, y = gx - ox, gy - oy
    bx, by = torch.floor(x), torch.floor(y)
    tx, ty = x - bx, y - by
    nodes, weights = [], []
    for j, wy in ((0, 1 - ty), (1, ty)):
        for i, wx in ((0, 1 - tx), (1, tx)):
            nodes.append((by.long() + j).clamp(0, h - 1) * w + (bx.long() + i).clamp(0, w - 1))
            weights.append(wx * wy)
    return nodes, weights, tx, ty


def _first_update(case, px, py, vx, vy):
    d, f64 = "cuda", torch.float64
    w, h, n = case["width"], case["height"], len(px)
    lanes = (n + 7) // 8 * 8
    dx32, dt = np.float32(case["cell"]), float(np.float32(case["dt"]))
    dx = float(dx32)
    # the sort: stable, by the Morton code of the cell that 32-bit positions give
    cell = [torch.from_numpy(np.clip((p / dx32), 0, m - 1).astype(np.int64)).to(d) for p, m in ((px, w), (py, h))]
    order = torch.argsort(_spread(cell[0]) | (_spread(cell[1]) << 1), stable=True)
    fluid = torch.zeros(h * w, dtype=torch.bool, device=d)
    fluid[cell[1] * w + cell[0]] = True
    fluid = fluid.view(h, w)
    del cell
    state = []
    for a in (px, py, vx, vy):
        b = torch.zeros(lanes, dtype=f64, device=d)
        b[:n] = torch.from_numpy(a).to(d).double()[order]
        state.append(b)
    px, py, vx, vy = state
    del order, state
    # particles to grid: momentum and weight on the faces, density on the cells
    wt = 0.75 ** 3 * 2.1875  # the temporal weight of a particle without a time residual
    gx, gy = px / dx, py / dx

    def scatter(ox, oy, sw, sh, value):
        sums = [torch.zeros(sw * sh, dtype=f64, device=d) for _ in range(2)]
        nodes, weights, _, _ = _corners(gx[:n], gy[:n], ox, oy, sw, sh)
        for node, wgt in zip(nodes, weights):
            sums[0].index_add_(0, node, wgt * wt)
            if value is not None:
                sums[1].index_add_(0, node, wgt * wt * value[:n])
        return [s.view(sh, sw) for s in sums]

    uw, um = scatter(0.0, 0.5, w + 1, h, vx)
    vw, vm = scatter(0.5, 0.0, w, h + 1, vy)
    dens = scatter(0.5, 0.5, w, h, None)[0]
    u, v = torch.where(uw > 0, um / uw, 0.0), torch.where(vw > 0, vm / vw, 0.0)
    u_ok, v_ok = uw > 0, vw > 0
    del um, vm, uw, vw
    solid = torch.zeros(h, w, dtype=torch.bool, device=d)
    solid[0], solid[-1], solid[:, 0], solid[:, -1] = True, True, True, True
    fluid &= ~solid
    near = torch.zeros(h + 1, w, dtype=torch.bool, device=d)
    near[1:] |= fluid
    near[:-1] |= fluid
    v = v + near * (GRAVITY * dt)
    # density smoothed over the fluid, then the pressure system
    sm, ff = dens, fluid.double()
    count = sum(_shift(ff, *s) for s in SIDES) + 4
    for _ in range(3):
        sm = torch.where(fluid, (4 * sm + sum(_shift(sm * ff, *s) for s in SIDES)) / count, dens)
    open_ = [~_shift(solid, *s, True) for s in SIDES]
    wet = [_shift(fluid, *s, False) for s in SIDES]
    div = (u[:, 1:] * open_[1] - u[:, :-1] * open_[0]) + (v[1:] * open_[3] - v[:-1] * open_[2])
    b = ff * (-div * dx + (sm - 9 * 1.15).clamp(0, 9) * 0.1 * dx * dx)
    diag = torch.zeros_like(b)
    for s, o, f in zip(SIDES, open_, wet):
        diag += o * torch.where(f, torch.ones_like(b), 1 / _theta(_shift(sm, *s), sm))
    diag = torch.where(fluid, diag, torch.ones_like(b))
    link = [(o & f & fluid).double() for o, f in zip(open_, wet)]
    del open_, wet, div, count

    def mul(p):
        q = diag * p
        for s, k in zip(SIDES, link):
            q -= k * _shift(p, *s)
        return q

    p, r = torch.zeros_like(b), b.clone()
    z = r / diag
    s_, rz, stop = z.clone(), (r * z).sum(), 1e-12 * b.norm()
    for it in range(20000 if bool(b.any()) else 0):
        q = mul(s_)
        alpha = rz / (s_ * q).sum()
        p += alpha * s_
        r -= alpha * q
        if it % 16 == 15 and bool(r.norm() <= stop):
            break
        z = r / diag
        new = (r * z).sum()
        s_ = z + (new / rz) * s_
        rz = new
    del r, z, s_, b, diag, link

    # projection, per face between cells `a` (left, below) and `c`
    def project(vel, ok, pa, pc, fa, fc, sa, sc, oa, oc):
        dp = torch.where(fa & fc, pc - pa, torch.where(fa, -pa / _theta(sc, sa), torch.where(
            fc, pc / _theta(sa, sc), torch.zeros_like(pa))))
        wall = oa != oc
        return torch.where(wall, torch.zeros_like(vel), vel - torch.where(oa, 0.0, dp) / dx), ok | wall

    def pair(a, axis, fill):
        lo = [1, 0, 0, 0] if axis else [0, 0, 1, 0]
        hi = [0, 1, 0, 0] if axis else [0, 0, 0, 1]
        return tuple(torch.nn.functional.pad(a, q, value=fill) for q in (lo, hi))

    def faces(vel, ok, axis):
        (pa, pc), (sa, sc) = pair(p, axis, 0.0), pair(sm, axis, 0.0)
        (fa, fc), (oa, oc) = pair(fluid, axis, False), pair(solid, axis, True)
        return project(vel, ok, pa, pc, fa, fc, sa, sc, oa, oc)

    u, u_ok = faces(u, u_ok, True)
    v, v_ok = faces(v, v_ok, False)
    for _ in range(4):
        for which in (0, 1):
            a, ok = (u, u_ok) if which == 0 else (v, v_ok)
            k = ok.double()
            cnt = sum(_shift(k, *s) for s in SIDES)
            mean = sum(_shift(a * k, *s) for s in SIDES) / cnt.clamp(min=1)
            a, ok = torch.where(ok | (cnt == 0), a, mean), ok | (cnt > 0)
            if which == 0:
                u, u_ok = a, ok
            else:
                v, v_ok = a, ok

    # grid to particles, over every lane of the last group of eight
    def gather(ox, oy, grid, opened):
        nodes, weights, _, _ = _corners(gx, gy, ox, oy, grid.shape[1], grid.shape[0])
        total, value = 0, 0
        for node, wgt in zip(nodes, weights):
            wgt = wgt * opened.reshape(-1)[node]
            total = total + wgt
            value = value + wgt * grid.reshape(-1)[node]
        return value / total.clamp(min=1e-6)

    left, right = pair(solid, True, True)
    below, above = pair(solid, False, True)
    nvx = gather(0.0, 0.5, u, (~(left | right)).double())
    nvy = gather(0.5, 0.0, v, (~(below | above)).double())
    m = torch.arange(lanes, device=d)
    for shift, mult in ((16, 0x7FEB352D), (15, 0x846CA68B), (16, 1)):
        m = ((m ^ (m >> shift)) * mult) & 0xFFFFFFFF
    jitter = (m & 0x7FFFFF).double() / (1 << 23) - 0.5
    scale = ((nvx * nvx + nvy * nvy).sqrt() * dt / dx).clamp(0, 1)
    act = (dt + scale * scale * (3 - 2 * scale) * jitter * dt).clamp(0, 2 * dt)
    out = []
    for at, vel, cells in ((px, nvx, w), (py, nvy, h)):
        low, high = 1.001 * dx, (cells - 1.001) * dx
        to = at + act * vel
        back = ((to < low) & (vel < 0)) | ((to > high) & (vel > 0))
        out.append((to.clamp(low, high), torch.where(back, -DAMPING * vel, vel)))

    def pack(x, y):
        return torch.stack([x.view(-1, 8), y.view(-1, 8)], 1).reshape(-1).cpu()

    return [pack(out[0][0], out[1][0]), pack(out[0][1], out[1][1])]
