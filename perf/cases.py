"""Workloads whose time a user of this framework waits for, through its public
entry points: frames of two substeps (a rendered frame at the default
dt = (1/60)/2) of dam-break scenes from a few thousand to millions of particles,
plain, adaptive and warm-started; the reference application's own loop; batches
of independent scenes; the host-buffer frame; a rendered image; a slice of
warm-start training; and the exclusive scan.

Every frame starts from a given device state (a roll-out, a co-simulation or a
slab exchange hands positions and velocities in and takes them out), so one pass
is upload, two substeps, download. The states are fluid columns in the middle of
their collapse: a lattice at half the kernel radius, compressed towards the
floor, spread along x, with the disorder of a moving fluid and a collapse
velocity field that vanishes at the walls.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from pbf_b200 import BatchSolver, Solver, autotune, learned, scenes
from pbf_b200 import solver as api
from pbf_b200._lib import check, lib
from pbf_b200.render import Renderer, box_camera

H = 0.1
DEV = "cuda"


def listed():
    return [
        # an interactive or control-loop scene: latency of every launch counts
        {"name": "frame_4k", "kind": "frame", "nx": 17, "ny": 16, "nz": 15, "cell": 0.5, "lanes": 2, "iters": 4},
        # the small dam break (32 a side) as a first-time user runs it: default cells and lanes
        {"name": "frame_33k", "kind": "frame", "nx": 32, "ny": 32, "nz": 32, "cell": 1.0, "lanes": 2, "iters": 4},
        # the headline dam break (64 a side) with the settings the autotuner picks
        {"name": "frame_262k", "kind": "frame", "nx": 64, "ny": 64, "nz": 64, "cell": 0.5, "lanes": 2, "iters": 4},
        # corrections until the density error is within 10 %, on a ragged block
        {"name": "adaptive_98k", "kind": "adaptive", "nx": 61, "ny": 39, "nz": 41, "cell": 0.5, "lanes": 2, "iters": 2,
         "tol": 0.1},
        # the learned warm start, two corrections (the fused feature and network pass)
        {"name": "warm_262k", "kind": "warm", "nx": 64, "ny": 64, "nz": 64, "cell": 0.5, "lanes": 2, "iters": 2},
        # the reference application: its scene 1 at its size and parameters, its three calls
        {"name": "app_262k", "kind": "app", "dim": 64},
        # many independent scenes in one handle (64 scenes of 4,096 to 65,536 particles)
        {"name": "batch_64", "kind": "batch", "scenes": 64, "lo": 4096, "hi": 65536, "counts": 0, "cell": 0.5},
        # the double dam break around a sphere with eight small scenes: 4.7 M particles
        {"name": "large_4700k", "kind": "large", "block": 128, "small": 65536, "scenes": 8, "cell": 0.5},
        # a renderer or co-simulation on the host: pinned buffers in, positions out
        {"name": "host_262k", "kind": "host", "nx": 64, "ny": 64, "nz": 64, "cell": 0.5, "lanes": 2, "iters": 4},
        # one image of the headline scene, read back
        {"name": "render_800", "kind": "render", "width": 800, "height": 800, "nx": 64, "ny": 64, "nz": 64},
        # sixteen Adam steps of the warm-start network and its weights
        {"name": "train_4096", "kind": "train", "batch": 4096, "steps": 16},
        # the scan on its own: cell counts of a large grid, a ragged length
        {"name": "scan_5m", "kind": "scan", "count": 5000001},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["frame"] * 5 + ["adaptive", "warm", "app", "batch", "batch", "large", "host", "render", "train",
                                       "scan"])
    if kind in ("frame", "adaptive", "warm", "host"):
        n = logint(4096, 1 << 20 if kind == "frame" else 300000)
        side = n ** (1.0 / 3.0)
        nx = max(4, int(side * rng.uniform(0.75, 1.35)))
        ny = max(4, int(side * rng.uniform(0.75, 1.35)))
        nz = max(4, int(round(n / (nx * ny))))
        c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "cell": rng.choice([0.5, 0.5, 1.0]),
             "lanes": rng.choice([1, 2, 2, 2, 4]), "iters": rng.choice([2, 3, 4, 4, 4, 6])}
        if kind == "adaptive":
            c.update(iters=2, tol=rng.choice([0.05, 0.1, 0.2]))
        if kind == "warm":
            c["iters"] = 2
        return c
    if kind == "app":
        return {"kind": "app", "dim": 2 * rng.randint(8, 32)}
    if kind == "batch":
        lo = logint(1000, 8192)
        return {"kind": "batch", "scenes": rng.randint(2, 64), "lo": lo, "hi": lo * rng.randint(2, 8),
                "counts": rng.randint(1, 1000), "cell": rng.choice([0.5, 1.0])}
    if kind == "large":
        return {"kind": "large", "block": rng.randint(72, 120), "small": logint(4096, 65536),
                "scenes": rng.randint(1, 8), "cell": rng.choice([0.5, 1.0])}
    if kind == "render":
        side = rng.randint(16, 64)
        return {"kind": "render", "width": rng.randint(320, 1280), "height": rng.randint(240, 800), "nx": side,
                "ny": side, "nz": side}
    if kind == "train":
        return {"kind": "train", "batch": rng.choice([1024, 2048, 4096, 8192]) - rng.choice([0, 0, 37]),
                "steps": rng.randint(4, 24)}
    return {"kind": "scan", "count": logint(30000, 20000000)}


# ---- inputs ----------------------------------------------------------------------
def column(nx, ny, nz, gen, origin=(0.05, 0.05, 0.05)):
    """Positions and velocities (float32 on the GPU) of a collapsing nx x ny x nz
    column whose lattice corner is at `origin` (x-fastest order)."""
    s = 0.5 * H
    i = torch.arange(nx * ny * nz, device=DEV)
    q = torch.stack([i % nx, (i // nx) % ny, i // (nx * ny)], 1).double()
    ext = torch.tensor([nx, ny, nz], dtype=torch.float64, device=DEV) * s
    u = q * s / ext                                   # 0 .. 1 inside the column
    p = q * s
    p[:, 1] *= 1.0 - 0.04 * (1.0 - u[:, 1])           # up to 4 % compressed towards the floor
    p[:, 0] *= 1.0 + 0.03 * (1.0 - u[:, 1])           # the foot spreads along x
    noise = 2.0 * torch.rand(p.shape, generator=gen, device=DEV, dtype=torch.float64) - 1.0
    p += 0.06 * H * noise
    v = torch.stack([1.5 * u[:, 0] * (1.0 - 0.5 * u[:, 1]), -1.5 * u[:, 1], 0.2 * (u[:, 2] - 0.5) * u[:, 1]], 1)
    v += 0.05 * u[:, 1:2] * (2.0 * torch.rand(p.shape, generator=gen, device=DEV, dtype=torch.float64) - 1.0)
    p += torch.tensor(origin, dtype=torch.float64, device=DEV)
    return p.float().contiguous(), v.float().contiguous()


def generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def box_of(cells):
    r = 0.3 * H
    box = [0.0, 0.0, 0.0, cells[0] * H, cells[1] * H, cells[2] * H]
    return box, [r, r, r, box[3] - r, box[4] - r, box[5] - r]


def column_cells(nx, ny, nz):
    """Grid cells of h: the column takes 0.4 x 0.8 x 0.8 of its box."""
    return (int(math.ceil(1.25 * nx)) + 1, int(math.ceil(0.625 * ny)) + 2, int(math.ceil(0.625 * nz)) + 2)


def scene_list(case, seed):
    """[(positions, velocities, cells, sphere)] of a case, in batch order."""
    g = generator(seed)
    none = (0.0, 0.0, 0.0, 0.0)
    if case["kind"] in ("frame", "adaptive", "warm", "host", "render"):
        n3 = (case["nx"], case["ny"], case["nz"])
        return [column(*n3, g) + (column_cells(*n3), none)]
    out = []
    if case["kind"] == "large":
        b = case["block"]
        cells = (int(2.5 * b), int(1.25 * b), int(1.25 * b))
        z0 = 0.5 * (cells[2] * H - 0.5 * H * b)
        p1, v1 = column(b, b, b, g, (0.05, 0.05, z0))
        p2, v2 = column(b, b, b, g, (0.05, 0.05, z0))
        p2, v2 = p2.clone(), v2.clone()
        p2[:, 0] = cells[0] * H - p2[:, 0]            # the second column falls the other way
        v2[:, 0] = -v2[:, 0]
        r = 0.15 * b * H
        out.append((torch.cat([p1, p2]), torch.cat([v1, v2]), cells, (0.5 * cells[0] * H, r, 0.5 * cells[2] * H, r)))
        counts = [case["small"]] * case["scenes"]
    else:
        rng = np.random.RandomState(case["counts"])
        counts = np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), case["scenes"])).round().astype(int)
    for c in counts:
        m = max(2, int(round(float(c) ** (1.0 / 3.0))))
        n3 = (m, m, int(math.ceil(c / (m * m))))
        p, v = column(*n3, g)
        out.append((p[:c].contiguous(), v[:c].contiguous(), column_cells(*n3), none))
    return out


def solver_of(case, sc):
    n = sum(int(s[0].shape[0]) for s in sc)
    para = scenes.benchmark_parameter(n, h=H, iterations=int(case.get("iters", 4)))
    ov = scenes.stable_overrides(para)
    ov.update(gravity=(0.0, -9.8, 0.0), cell_scale=case["cell"], pair_lanes=case.get("lanes", 2), block_size=256)
    if case["kind"] == "adaptive":
        ov.update(adaptive=1, density_tol=case["tol"], max_iterations=32)
    if case["kind"] == "warm":
        ov.update(warm_start=1, warm_clamp=4.0, warm_floor=1)
    if len(sc) == 1 and case["kind"] not in ("batch", "large"):
        box, bd = box_of(sc[0][2])
        return Solver(para, box, bd, api.default_ext(grid_dims=autotune.dims_for_scale(sc[0][2], case["cell"]), **ov))
    descs = []
    for p, _, cells, sphere in sc:
        box, bd = box_of(cells)
        descs.append({"grid_space": box, "boundary": bd, "grid_dims": autotune.dims_for_scale(cells, case["cell"]),
                      "nparticles": int(p.shape[0]), "sphere": sphere})
    return BatchSolver(para, descs, api.default_ext(**ov))


def warm_network(seed):
    """A warm-start network from the seed: random hidden layers and a read-out
    that follows the previous substep's total lambda and the density (the two
    features a trained network leans on), as BF16 weights and constants."""
    w, b = learned.init_params(seed)
    b[learned.FMEAN:learned.FMEAN + 12] = [0.5, 1.0, -1e-4, 200.0, 0.0, 4.0, 4.0, 4.0, 0.1, 0.1, 0.2, 0.1]
    b[learned.FISTD:learned.FISTD + 12] = [8.0, 8.0, 5e3, 0.01, 0.1, 1.0, 1.0, 1.0, 10.0, 5.0, 2.0, 5.0]
    b[learned.OSCALE] = 2e-4
    return learned.bf16_bits(w), b


def train_rows(case, seed):
    g = generator(seed)
    n = case["batch"] * case["steps"]
    f = torch.randn((n, 12), generator=g, device=DEV)
    f = f * torch.linspace(0.2, 2.0, 12, device=DEV) + torch.linspace(-1.0, 1.0, 12, device=DEV)
    t = 1e-3 * (torch.tanh(f[:, 2]) - 0.5 * f[:, 1] + 0.2 * f[:, 3] * f[:, 0])
    return f.contiguous(), t.contiguous()


TRAIN_LR = 2e-3


# ---- one pass --------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("frame", "adaptive", "warm", "batch", "large", "host"):
        sc = scene_list(case, seed)
        st["pos"] = torch.cat([s[0] for s in sc])
        st["vel"] = torch.cat([s[1] for s in sc])
        st["solver"] = solver_of(case, sc)
        if kind == "warm":
            learned.install(st["solver"], *warm_network(seed))
        if kind == "host":
            st["pos"] = st["pos"].cpu().pin_memory()
            st["vel"] = st["vel"].cpu().pin_memory()
            st["out"] = torch.empty_like(st["pos"]).pin_memory()
        else:
            st["opos"] = torch.empty_like(st["pos"])
            st["ovel"] = torch.empty_like(st["vel"])
    elif kind == "app":
        sc = scenes.reference_app_scene(1, seed=int(seed) % (1 << 32), dims=(case["dim"],) * 3)
        s = api.initCUDASolverDataBuffer(sc.pos, sc.vel, sc.para, sc.grid_space, sc.boundary, sc.ext())
        st.update(solver=s, para=sc.para, pos=torch.from_numpy(sc.pos).to(DEV), vel=torch.from_numpy(sc.vel).to(DEV))
        st["shown"] = torch.empty_like(st["pos"])
        st["ovel"] = torch.empty_like(st["vel"])
        s.bind_position(st["shown"])
    elif kind == "render":
        p, _, cells, _ = scene_list(case, seed)[0]
        box, _ = box_of(cells)
        st["pos"] = p
        st["cam"] = box_camera(box, case["width"], case["height"], 0.3 * H)
        st["renderer"] = Renderer(case["width"], case["height"])
    elif kind == "train":
        f, t = train_rows(case, seed)
        w, b = learned.init_params(seed % 1000)
        b = learned.set_normalisation(b, f.cpu().numpy(), t.cpu().numpy())
        st.update(feat=f, target=t, trainer=learned.Trainer(w, b, max_batch=case["batch"]))
    else:
        g = generator(seed)
        m = case["count"]
        st["counts"] = torch.randint(0, 12, (m,), generator=g, device=DEV, dtype=torch.int32)
        st["out"] = torch.empty(m + 1, dtype=torch.int32, device=DEV)
        st["bytes"] = int(lib().pbf_scan_workspace_bytes(m))
        st["ws"] = torch.empty(st["bytes"], dtype=torch.uint8, device=DEV)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    stream = torch.cuda.current_stream()
    if kind in ("frame", "adaptive", "warm", "batch", "large"):
        s = st["solver"]
        s.upload_device(st["pos"], st["vel"], stream)
        s.step(2, stream)
        s.download_device(st["opos"], st["ovel"], stream)
        return {"pos": st["opos"], "vel": st["ovel"]}
    if kind == "host":
        st["solver"].step_host(st["pos"], st["vel"], st["out"], 2, stream)
        return {"pos": st["out"]}
    if kind == "app":
        s = st["solver"]
        s.upload_device(st["pos"], st["vel"], None)
        for _ in range(2):
            api.cudaPBFSolve(s, st["para"])
        s.download_device(None, st["ovel"], None)
        return {"pos": st["shown"], "vel": st["ovel"]}
    if kind == "render":
        st["renderer"].frame(st["cam"], positions=st["pos"], stream=stream)
        return {"color": st["renderer"].read("color")}
    if kind == "train":
        b = case["batch"]
        for i in range(case["steps"]):
            st["trainer"].step(st["feat"][i * b:(i + 1) * b], st["target"][i * b:(i + 1) * b], TRAIN_LR)
        w, bias, _ = st["trainer"].params()
        return {"weights": w, "biases": bias}
    check(lib().pbf_scan_exclusive_i32(st["counts"].data_ptr(), st["out"].data_ptr(), case["count"],
                                       st["ws"].data_ptr(), C.c_size_t(st["bytes"]), int(stream.cuda_stream)))
    return {"starts": st["out"]}


# ---- what a pass cannot do without -------------------------------------------------
PAIRS = 33  # neighbours of an interior particle at rest spacing


def work(case):
    kind = case["kind"]
    if kind == "train":
        rows = case["batch"] * case["steps"]
        mac = 12 * 64 + 2 * 64 * 64 + 64
        return {"bytes": 52.0 * rows + 4.0 * 2 * 9506, "flops": 6.0 * mac * rows}
    if kind == "scan":
        return {"bytes": 8.0 * case["count"], "flops": float(case["count"])}
    if kind == "render":
        px = case["width"] * case["height"]
        return {"bytes": 12.0 * case["nx"] * case["ny"] * case["nz"] + 16.0 * px, "flops": 60.0 * 70.0 * px}
    if kind == "app":
        n, iters = case["dim"] ** 3, 4
    elif kind == "batch":
        rng = np.random.RandomState(case["counts"])
        c = np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"]), case["scenes"])).round()
        n, iters = float(c.sum()), 4
    elif kind == "large":
        n, iters = 2 * case["block"] ** 3 + case["scenes"] * case["small"], 4
    else:
        n, iters = case["nx"] * case["ny"] * case["nz"], case["iters"]
    io = 36.0 if kind == "host" else 48.0
    # 30 flops a pair for the density and its gradient, 40 for the correction, 25 for the
    # curl and 30 for the vorticity and viscosity
    return {"bytes": io * n, "flops": 2.0 * n * PAIRS * (70.0 * iters + 55.0)}


# ---- the same in 64 bits -----------------------------------------------------------
def exact(case, seed):
    """Plain torch in 64 bits. None for the scan (whole numbers), and for the
    image: which sprite covers a silhouette's texel is a decision in 32 bits."""
    kind = case["kind"]
    if kind in ("scan", "render"):
        return None
    if kind == "train":
        return exact_train(case, seed)
    if kind == "app":
        s = scenes.reference_app_scene(1, seed=int(seed) % (1 << 32), dims=(case["dim"],) * 3)
        sc = [(torch.from_numpy(s.pos).to(DEV), torch.from_numpy(s.vel).to(DEV), (64, 64, 64), (0.0,) * 4)]
        f = Fluid(sc, s.para, s.ext(), [(s.grid_space, s.boundary)])
    else:
        sc = scene_list(case, seed)
        n = sum(int(s[0].shape[0]) for s in sc)
        para = scenes.benchmark_parameter(n, h=H, iterations=int(case.get("iters", 4)))
        ov = scenes.stable_overrides(para)
        f = Fluid(sc, para, api.default_ext(gravity=(0.0, -9.8, 0.0), **ov), [box_of(s[2]) for s in sc])
    if kind == "adaptive":
        f.adapt = (case["tol"], 32)
    if kind == "warm":
        f.net = warm_network(seed)
    for _ in range(2):
        f.substep()
    if kind == "host":
        return {"pos": f.x.cpu()}
    return {"pos": f.x, "vel": f.v}


class Fluid:
    """Position Based Fluids in float64 over a list of neighbour pairs."""

    def __init__(self, sc, para, ext, boxes):
        self.x = torch.cat([s[0] for s in sc]).double()
        self.v = torch.cat([s[1] for s in sc]).double()
        self.sid = torch.cat([torch.full((s[0].shape[0],), i, device=DEV) for i, s in enumerate(sc)])
        t = lambda rows: torch.tensor(rows, dtype=torch.float64, device=DEV)  # noqa: E731
        f32 = lambda rows: t(np.asarray(rows, np.float32).astype(np.float64))  # noqa: E731
        self.gmin = f32([b[0][:3] for b in boxes])[self.sid]
        self.bmin = f32([b[1][:3] for b in boxes])[self.sid]
        self.bmax = f32([b[1][3:] for b in boxes])[self.sid]
        self.sphere = f32([s[3] for s in sc])[self.sid]
        self.p, self.e = para, ext
        self.h = float(para.h)
        self.adapt = self.net = None
        self.total = torch.zeros_like(self.x[:, 0])

    def bound(self, x):
        def offset(u, w):
            a = torch.sin(2.0 * (u * 12.9898 + w * 78.233)) * 43758.5453
            return (a - torch.trunc(a)).abs() * float(self.e.wall_jitter)
        for a, lo, hi in ((0, (1, 2), (1, 2)), (1, (0, 2), (1, 2)), (2, (0, 1), (0, 1))):
            x[:, a] = torch.where(x[:, a] < self.bmin[:, a], self.bmin[:, a] + offset(x[:, lo[0]], x[:, lo[1]]), x[:, a])
            x[:, a] = torch.where(x[:, a] > self.bmax[:, a], self.bmax[:, a] - offset(x[:, hi[0]], x[:, hi[1]]), x[:, a])
        d = x - self.sphere[:, :3]
        r = self.sphere[:, 3]
        l = d.norm(dim=1)
        inside = (r > 0) & (l < r) & (l > 0)
        return torch.where(inside[:, None], self.sphere[:, :3] + d * (r / l.clamp_min(1e-30))[:, None], x)

    def search(self, x):
        """Pairs (i, j), i != j, within h: cells of h, 27 cells around each particle."""
        c = torch.floor((x - self.gmin) / self.h).long() + 2
        span = int(c.max()) + 3
        key = ((self.sid * span + c[:, 2]) * span + c[:, 1]) * span + c[:, 0]
        order = torch.argsort(key)
        sk = key[order]
        ii, jj = [], []
        step = 1 << 18
        for b in range(0, x.shape[0], step):
            k0 = key[b:b + step]
            me = torch.arange(b, b + k0.shape[0], device=DEV)
            for dz in (-1, 0, 1):
                for dy in (-1, 0, 1):
                    row = k0 + (dz * span + dy) * span
                    lo = torch.searchsorted(sk, row - 1)
                    cnt = torch.searchsorted(sk, row + 2) - lo
                    i = torch.repeat_interleave(me, cnt)
                    first = torch.repeat_interleave(lo - (torch.cumsum(cnt, 0) - cnt), cnt)
                    j = order[first + torch.arange(i.shape[0], device=DEV)]
                    keep = (i != j) & (((x[i] - x[j]) ** 2).sum(1) <= self.h * self.h)
                    ii.append(i[keep])
                    jj.append(j[keep])
        return torch.cat(ii), torch.cat(jj)

    def add(self, i, v):
        return torch.zeros((self.x.shape[0],) + v.shape[1:], dtype=torch.float64, device=DEV).index_add_(0, i, v)

    def pairs(self, x, i, j):
        h = self.h
        r = x[i] - x[j]
        r2 = (r * r).sum(1)
        t = (h * h - r2).clamp_min(0.0)
        w = 315.0 * 0.31830988618 / (64.0 * h ** 9) * t ** 3
        l = r2.sqrt()
        g = torch.where((l <= h) & (l >= float(self.e.grad_rmin)),
                        -45.0 * 0.31830988618 / h ** 6 * (h - l) ** 2 / l.clamp_min(1e-30), torch.zeros_like(l))
        return r, w, g[:, None] * r

    def wall(self, x):
        rho = torch.zeros_like(x[:, 0])
        g = torch.zeros_like(x)
        if not (self.e.flags & 4):
            return rho, g
        h = self.h
        n = float(self.p.restRho) + 315.0 * 0.31830988618 / (64.0 * h ** 9) * h ** 6
        for a in range(3):
            for d, sign in ((x[:, a] - self.bmin[:, a], 1.0), (self.bmax[:, a] - x[:, a], -1.0)):
                s = d.clamp_min(0.0) / h
                f = 0.5 - 315.0 / 256.0 * (s - 4 / 3 * s ** 3 + 6 / 5 * s ** 5 - 4 / 7 * s ** 7 + s ** 9 / 9)
                near = d < h
                rho += torch.where(near, n * f, torch.zeros_like(f))
                g[:, a] += torch.where(near, -sign * n * 315.0 / (256.0 * h) * (1 - s * s) ** 4, torch.zeros_like(f))
        return rho, g

    def lam(self, x, i, j):
        """lambda, the largest one-sided density error, and what the features need."""
        rho0 = float(self.p.restRho)
        r, w, g = self.pairs(x, i, j)
        rho = self.add(i, w)
        gs = self.add(i, g)
        gw = gs.norm(dim=1)
        err = float((rho / rho0 - 1.0).clamp_min(0.0).max())
        fluid = rho / rho0
        rw, gg = self.wall(x)
        c = (rho + rw) / rho0 - 1.0
        if self.e.flags & 1:
            c = c.clamp_min(0.0)
        gs = gs + gg
        den = (self.add(i, (g * g).sum(1)) + (gs * gs).sum(1)) / rho0 ** 2
        return -c / (den + float(self.p.epsilon)), err, (r, g, den, fluid, gw)

    def correct(self, x, lam, i, j):
        p, e = self.p, self.e
        _, w, g = self.pairs(x, i, j)
        wq = 315.0 * 0.31830988618 / (64.0 * self.h ** 9) * (self.h ** 2 - float(p.deltaq) ** 2) ** 3
        s = lam[i] + lam[j] - float(p.k) * (w / wq) ** float(p.n) * float(e.scorr_scale)
        a = self.add(i, s[:, None] * g)
        if e.flags & 4:
            a = a + lam[:, None] * self.wall(x)[1]
        return self.bound(x + a / float(p.restRho))

    def warm(self, x, v, lam, i, j, more):
        """lambda0 of the network, clamped to the trust region (floor 1, clamp 4)."""
        r, g, den, fluid, gw = more
        h, rho0 = self.h, float(self.p.restRho)
        cap = float(self.e.max_neighbors)
        dv = v[j] - v[i]
        one = torch.ones_like(i, dtype=torch.float64)
        cnt = self.add(i, one)
        near = torch.minimum(x - self.bmin, self.bmax - x).div(h).clamp(0.0, 4.0)
        f = torch.stack([cnt / cap, fluid, self.total, den, self.add(i, (dv * g).sum(1)) / rho0, near[:, 0],
                         near[:, 1], near[:, 2], self.add(i, ((r * r).sum(1) < 0.25 * h * h).double()) / cap,
                         self.add(i, r).norm(dim=1) / h / cnt.clamp_min(1.0), gw * h / rho0,
                         self.add(i, (dv * dv).sum(1)) * (float(self.p.dt) / h) ** 2 / cnt.clamp_min(1.0)], 1)
        w16, b = self.net
        w = torch.from_numpy((w16.astype(np.uint32) << 16).view(np.float32).astype(np.float64)).to(DEV)
        b = torch.from_numpy(np.asarray(b, np.float64)).to(DEV)
        a = (f - b[learned.FMEAN:learned.FMEAN + 12]) * b[learned.FISTD:learned.FISTD + 12]
        w1 = w[learned.W1:learned.W2].view(64, 16)[:, :12]
        for wl, bl in ((w1, b[0:64]), (w[learned.W2:learned.W3].view(64, 64), b[64:128]),
                       (w[learned.W3:learned.W4].view(64, 64), b[128:192])):
            a = torch.nn.functional.gelu(a @ wl.t() + bl, approximate="tanh")
        y = (a @ w[learned.W4:] + b[learned.B4]) * b[learned.OSCALE]
        return torch.maximum(torch.minimum(y, torch.maximum(lam, 4.0 * lam)), torch.minimum(lam, 4.0 * lam))

    def substep(self):
        p = self.p
        dt, rho0 = float(p.dt), float(p.restRho)
        g = torch.tensor([float(a) for a in self.e.gravity], dtype=torch.float64, device=DEV)
        old = self.x
        v = self.v + dt * g
        x = self.bound(old + dt * v)
        i, j = self.search(x)
        total = torch.zeros_like(self.total)
        k = 0
        while True:
            lam, err, more = self.lam(x, i, j)
            if k >= int(p.iterations) and (self.adapt is None or err <= self.adapt[0] or k >= self.adapt[1]):
                break
            if self.net is not None and k == 0:
                lam = self.warm(x, v, lam, i, j, more)
            total = total + lam
            x = self.correct(x, lam, i, j)
            k += 1
        self.total = total
        v = (x - old) / dt
        _, w, gr = self.pairs(x, i, j)
        dv = v[j] - v[i]
        om = self.add(i, torch.cross(dv, gr, dim=1))
        eta = self.add(i, om.norm(dim=1)[j][:, None] * gr)
        l = eta.norm(dim=1, keepdim=True)
        eta = torch.where(l > 1e-3, eta / l.clamp_min(1e-30), eta)
        visc = float(p.c) / (rho0 if self.e.flags & 2 else 1.0)
        dvel = dt * float(p.vorticityConfinementEpilon) * torch.cross(eta, om, dim=1) + visc * self.add(i, dv * w[:, None])
        self.x, self.v = x, v + dvel


def exact_train(case, seed):
    """The Adam steps in float64 (BF16 weights in the products, as the trainer rounds them)."""
    f, t = train_rows(case, seed)
    w, b = learned.init_params(seed % 1000)
    b = learned.set_normalisation(b, f.cpu().numpy(), t.cpu().numpy())
    w = torch.from_numpy(w.astype(np.float64)).to(DEV)
    b = torch.from_numpy(b.astype(np.float64)).to(DEV)
    nb = learned.B4 + 1
    mean, istd = b[learned.FMEAN:learned.FMEAN + 12], b[learned.FISTD:learned.FISTD + 12]
    m = [torch.zeros_like(w), torch.zeros_like(b[:nb])]
    s = [torch.zeros_like(w), torch.zeros_like(b[:nb])]
    rows = case["batch"]
    for k in range(case["steps"]):
        x = (f[k * rows:(k + 1) * rows].double() - mean) * istd
        y = t[k * rows:(k + 1) * rows].double() / b[learned.OSCALE]
        wr = w.to(torch.bfloat16).double().requires_grad_(True)
        br = b[:nb].clone().requires_grad_(True)
        a = x
        for wl, bl in ((wr[learned.W1:learned.W2].view(64, 16)[:, :12], br[0:64]),
                       (wr[learned.W2:learned.W3].view(64, 64), br[64:128]),
                       (wr[learned.W3:learned.W4].view(64, 64), br[128:192])):
            a = torch.nn.functional.gelu(a @ wl.t() + bl, approximate="tanh")
        loss = ((a @ wr[learned.W4:] + br[learned.B4] - y) ** 2).mean()
        gw, gb = torch.autograd.grad(loss, (wr, br))
        for p, g, q in ((w, gw, 0), (b[:nb], gb, 1)):
            m[q] = 0.9 * m[q] + 0.1 * g
            s[q] = 0.999 * s[q] + 0.001 * g * g
            p -= TRAIN_LR * (m[q] / (1 - 0.9 ** (k + 1))) / ((s[q] / (1 - 0.999 ** (k + 1))).sqrt() + 1e-8)
    return {"weights": w.cpu(), "biases": b.cpu()}
