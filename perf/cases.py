"""The workloads this framework's speed is measured on.

A case is one call, or one short sequence of calls, that a program using the
simulator makes again and again:

  frames    whole time steps (`bubblesim`) of a benchmark configuration, with
            the surfaces a renderer takes after each pass
  project   the grid velocity update of one step on its own: particle-to-grid
            transfer, wall rules, pressure projection
  levelset  signed distances and cell marks from the particles
  surface   marching-cubes extraction of the liquid and gas surfaces
  gradient  loss and gradient through recorded steps (the adjoint)

Grids run from 32^3 to 256^3, cubic and ragged, in the mixed and the all-FP64
form of the projection. `listed()` names the cases, `draw()` gives more of the
same ranges, `prepare()` makes what a program has in hand before the call and
`run()` makes the call and returns what it computed.
"""
from __future__ import annotations

import ctypes as C
import importlib

import numpy as np
import torch

mp = importlib.import_module("2017multiphase_b200")

LEVEL = 0.8          # liquid height of the bubble column, as a share of the box


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest simulation in use: previews and parameter searches run
        # thousands of these; bound by launches, host round trips and latency
        {"name": "frames_bubble_32", "kind": "frames", "config": 1, "n": 32, "frames": 4, "restore": True},
        # pool boiling: heat, gas generation and phase change in every step
        {"name": "frames_boil_64", "kind": "frames", "config": 2, "n": 64, "frames": 4, "restore": True},
        # melting and freezing: solid particles, their surface and a heat solve
        {"name": "frames_melt_96", "kind": "frames", "config": 3, "n": 96, "frames": 2, "restore": False},
        # the production size: 256^3, ~105M particles, surfaces every step
        {"name": "frame_column_256", "kind": "frames", "config": 5, "n": 256, "frames": 1, "restore": False},
        # the projection by itself, as a host application with its own
        # advection calls it: small, ragged, in FP64, and large
        {"name": "project_64", "kind": "project", "nx": 64, "ny": 64, "nz": 64, "precision": "mixed"},
        {"name": "project_90x66x110", "kind": "project", "nx": 90, "ny": 66, "nz": 110, "precision": "mixed"},
        {"name": "project_fp64_96", "kind": "project", "nx": 96, "ny": 96, "nz": 96, "precision": "fp64"},
        {"name": "project_256", "kind": "project", "nx": 256, "ny": 256, "nz": 256, "precision": "mixed"},
        # distances and marks for a renderer or a coupling code
        {"name": "levelset_128", "kind": "levelset", "nx": 128, "ny": 128, "nz": 128},
        # surfaces of a stored particle set
        {"name": "surface_128x96x144", "kind": "surface", "nx": 128, "ny": 96, "nz": 144},
        # one iteration of an optimisation over initial velocities
        {"name": "gradient_dam_64", "kind": "gradient", "config": 4, "n": 64, "steps": 8},
        # sensitivity of the two-phase flow at its recorded state
        {"name": "gradient_column_96", "kind": "gradient", "config": 5, "n": 96, "steps": 4},
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm of lo..hi, odd ones among them."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["frames", "frames", "project", "project", "levelset", "surface", "gradient"])
    if kind == "frames":
        config = rng.choice([1, 2, 3, 5])
        if config in (1, 2):
            return {"kind": kind, "config": config, "n": _size(rng, 24, 72), "frames": rng.choice([2, 4]),
                    "restore": True}
        if config == 3:
            return {"kind": kind, "config": config, "n": _size(rng, 40, 100), "frames": 2, "restore": False}
        return {"kind": kind, "config": config, "n": _size(rng, 48, 200), "frames": 1, "restore": False}
    if kind == "gradient":
        if rng.random() < 0.5:
            return {"kind": kind, "config": 4, "n": _size(rng, 24, 64), "steps": rng.choice([4, 8])}
        return {"kind": kind, "config": 5, "n": _size(rng, 32, 96), "steps": rng.choice([2, 4])}
    base = _size(rng, 32, 160)
    case = {"kind": kind}
    for axis in ("nx", "ny", "nz"):
        # one grid in three is cubic; the others have three sizes of their own
        case[axis] = base
    if rng.random() < 0.67:
        for axis in ("nx", "ny", "nz"):
            case[axis] = max(24, min(200, int(base * (0.7 + 0.6 * rng.random()))))
    if kind == "project":
        case["precision"] = "fp64" if base <= 100 and rng.random() < 0.25 else "mixed"
    return case


# ---------------------------------------------------------------------------
# inputs, on the GPU from the seed
# ---------------------------------------------------------------------------
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _spheres(seed, dims, h):
    """Bubbles of the column as (x, y, z, r): radii of 1 to 4 % of the box, but
    a bubble is at least two cells wide, as the column's are on fine grids."""
    rng = np.random.default_rng(seed)
    box = np.asarray(dims, np.float64) * h
    r = np.maximum(rng.uniform(0.01, 0.04, 200) * box.min(), 1.5 * h)
    lo = 2 * h + r
    c = [lo + (ext - 2 * h - r - lo) * rng.random(200) for ext in (box[0], box[1], LEVEL * box[2])]
    return np.stack(c + [r], 1)


def _ball(sphere, dims, h):
    """The block of cells that a sphere touches, as three slices."""
    out = []
    for a in range(3):
        lo = max(0, int((sphere[a] - sphere[3]) / h) - 1)
        out.append(slice(lo, min(dims[a], int((sphere[a] + sphere[3]) / h) + 2)))
    return tuple(out)


def _lattice(p, g, right, top):
    """Positions (right, ny - 2, top, 8, 3) of a block of liquid in the corner
    of the grid of `p`: eight particles per cell, one in each eighth of the
    cell at a uniform position, as the framework's configurations have them."""
    h = p.cellsize
    shape = (right, p.ny - 2, top, 8)
    pos = torch.empty(shape + (3,), device="cuda")
    pos.uniform_(0.001, 0.999, generator=g)
    q = torch.arange(8, device="cuda")
    for a in range(3):
        cell = torch.arange(1, shape[a] + 1, device="cuda", dtype=torch.float32)
        view = [1, 1, 1, 1]
        view[a] = -1
        v = pos[..., a]
        v.add_(((q >> a) & 1).float()).mul_(0.5).add_(cell.view(view)).mul_(h)
    return pos


def _dam_particles(p, seed):
    """The dam break's block of liquid (x < 0.4, z < 0.6 of the box, in whole
    cells) with velocities N(0, 0.1)."""
    g = _generator(seed)
    pos = _lattice(p, g, int(0.4 * p.nx), int(0.6 * p.nz)).reshape(-1, 3)
    vel = torch.empty_like(pos).normal_(0.0, 0.1, generator=g)
    return pos, vel, torch.full((len(pos),), mp.TYPEFLUID, dtype=torch.int8, device="cuda")


def _column_particles(p, seed):
    """Particles of the bubble column on the grid of `p`: liquid up to its
    level, AIR inside the bubbles; a smooth swirl plus small fluctuations."""
    dims, h = (p.nx, p.ny, p.nz), p.cellsize
    g = _generator(seed)
    pos = _lattice(p, g, p.nx - 2, min(p.nz - 2, int(LEVEL * p.nz)))
    flag = torch.full(pos.shape[:-1], mp.TYPEFLUID, dtype=torch.int8, device="cuda")
    for s in _spheres(seed, dims, h):
        b = tuple(slice(max(0, t.start - 1), max(0, t.stop - 1)) for t in _ball(s, dims, h))
        d = pos[b] - torch.tensor(s[:3], device="cuda", dtype=torch.float32)
        flag[b][(d * d).sum(-1) < float(s[3]) ** 2] = mp.TYPEAIR
    pos, flag = pos.reshape(-1, 3), flag.reshape(-1)
    ph = torch.rand(3, 3, generator=g, device="cuda") * 6.2831853
    vel = torch.empty_like(pos).normal_(0.0, 0.02, generator=g)
    two_pi = 6.2831853 / (h * min(dims))
    for a in range(3):
        for b in range(3):
            if a != b:
                vel[:, a] += 0.2 * torch.sin(two_pi * pos[:, b] + ph[a, b])
    return pos, vel, flag


def _column_params(nx, ny, nz, config=5):
    p = mp.scene_params(config, max(nx, ny, nz))
    p.nx, p.ny, p.nz = nx, ny, nz
    p.par_num_max = 8 * (nx - 2) * (ny - 2) * (nz - 2) + 4096
    share = nx * ny * nz / 256.0 ** 3
    p.mc_max_verts = int(max(1 << 20, 64000000 * share))
    p.mc_max_tris = 2 * p.mc_max_verts
    return p


def _sim(p, pos, vel, flag):
    sim = mp.Sim(p)
    mass = np.full(flag.numel(), p.m0, np.float32)
    sim.upload_particles(pos.cpu().numpy(), flag.cpu().numpy(), mass, vel=vel.cpu().numpy(),
                         temp=None, lheat=None, solubility=None, gascontain=None)
    sim.set_tables(np.random.default_rng(1).random(10000, dtype=np.float32), np.zeros(0, np.int32))
    return sim


def _cell_marks(p, seed):
    """Marks and merged level set of the column's geometry at the cell centres
    (negative in the liquid, positive in the bubbles), float32."""
    dims, h = (p.nx, p.ny, p.nz), p.cellsize
    centre = [(torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) * h for n in dims]
    x, y, z = torch.meshgrid(*centre, indexing="ij")
    ls = torch.full(dims, -5.0 * h, dtype=torch.float64, device="cuda")
    for s in _spheres(seed, dims, h):
        b = _ball((s[0], s[1], s[2], s[3] + 5 * h), dims, h)
        d = float(s[3]) - torch.sqrt((x[b] - s[0]) ** 2 + (y[b] - s[1]) ** 2 + (z[b] - s[2]) ** 2)
        ls[b] = torch.maximum(ls[b], torch.clamp(d, -5.0 * h, 5.0 * h))
    mark = torch.where(ls > 0, mp.TYPEAIR, mp.TYPEFLUID).to(torch.int8)
    mark[:, :, 1 + min(p.nz - 2, int(LEVEL * p.nz)):] = mp.TYPEVACUUM
    for a in range(3):
        mark.select(a, 0).fill_(mp.TYPEBOUNDARY)
        mark.select(a, dims[a] - 1).fill_(mp.TYPEBOUNDARY)
    return mark, ls.float()


def _pinned_zeros(count, dtype):
    return torch.zeros(count, dtype=dtype).pin_memory()


class Meshes:
    """Page-locked host buffers that the surfaces of one simulation land in,
    sized once for the grid; a surface fills their front part."""

    def __init__(self, p, surfaces):
        self.nv = 40 * max(p.nx * p.ny, p.ny * p.nz, p.nx * p.nz) + 60000
        self.ni = 6 * self.nv
        self.buf = {s: (_pinned_zeros(3 * self.nv, torch.float32), _pinned_zeros(3 * self.nv, torch.float32),
                        _pinned_zeros(self.ni, torch.int32)) for s in surfaces}

    def take(self, sim):
        st = sim.state()
        out = {}
        for s, (v, n, i) in self.buf.items():
            mp._check(sim.lib.mp_mc_download(sim.ctx, s, v.data_ptr(), n.data_ptr(), i.data_ptr(), self.nv, self.ni),
                      sim.ctx)
            out["surface%d" % s] = [v, n, i, st.mc_verts[s], st.mc_indices[s]]
        return out


class Particles:
    """Page-locked host buffers for all particles, sized for the simulation's
    capacity; the particles there are now fill their front part."""

    def __init__(self, p):
        cap = p.par_num_max
        self.buf = [_pinned_zeros(3 * cap, torch.float32), _pinned_zeros(3 * cap, torch.float32),
                    _pinned_zeros(cap, torch.int8)] + [_pinned_zeros(cap, torch.float32) for _ in range(5)]

    def take(self, sim):
        count = C.c_int()
        mp._check(sim.lib.mp_download_particles(sim.ctx, C.byref(count), *[t.data_ptr() for t in self.buf]), sim.ctx)
        return self.buf + [count.value]


class Fields:
    """Page-locked host buffers for grid fields."""

    def __init__(self, sim, names):
        self.buf = {}
        for nm in names:
            cnt, eb = sim.field_info(nm)
            self.buf[nm] = _pinned_zeros(cnt, torch.int8 if eb == 1 else torch.float32)

    def take(self, sim):
        for nm, t in self.buf.items():
            mp._check(sim.lib.mp_get_field(sim.ctx, mp.FIELD_ID[nm], C.c_void_p(t.data_ptr()),
                                           t.numel() * t.element_size()), sim.ctx)
        return dict(self.buf)


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
PROJECT_FIELDS = ["press", "waterux", "wateruy", "wateruz"]
LEVELSET_FIELDS = ["lsmerge", "lsfluid", "lsair", "mark"]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "frames":
        if case["config"] == 5:
            p = _column_params(case["n"], case["n"], case["n"])
            sim = _sim(p, *_column_particles(p, seed))
        else:
            sim = mp.Sim.from_config(case["config"], case["n"], seed)
        surfaces = [mp.MC_FLUID, mp.MC_GAS] + ([mp.MC_SOLID] if case["config"] == 3 else [])
        s = {"kind": kind, "sim": sim, "frames": case["frames"], "meshes": Meshes(sim.params, surfaces)}
        s["start"] = sim.checkpoint() if case["restore"] else None
        s["particles"] = Particles(sim.params) if case["restore"] else None
        return s
    if kind == "gradient":
        if case["config"] == 4:
            p = mp.scene_params(4, case["n"])
            sim = _sim(p, *_dam_particles(p, seed))
            height = 0.3
        else:
            p = _column_params(case["n"], case["n"], case["n"])
            p.b_correct_position, p.b_run_mc = 0, 0
            sim = _sim(p, *_column_particles(p, seed))
            height = 0.7
        vel = torch.from_numpy(sim.download_particles()["vel"]).cuda().double()
        sim.adj_record(case["steps"], case["steps"])
        sim.adj_set_targets(mp.dam_break_targets(4096, seed, height=height))
        s = {"kind": kind, "sim": sim, "v0": None}
        if case["config"] == 4:
            # velocities a little away from the recorded ones, as after a
            # step of the optimiser
            vel += 1e-3 * torch.randn(vel.shape, generator=_generator(seed), device="cuda", dtype=torch.float64)
            s["v0"] = vel.requires_grad_()
        return s
    p = _column_params(case["nx"], case["ny"], case["nz"])
    p.b_run_mc = 1 if kind == "surface" else 0
    if kind == "project" and case["precision"] == "fp64":
        p.precision = mp.PREC_FP64
    sim = _sim(p, *_column_particles(p, seed))
    s = {"kind": kind, "sim": sim}
    if kind == "surface":
        s["meshes"] = Meshes(p, [mp.MC_FLUID, mp.MC_GAS])
        return s
    sim.hashAndSortParticles()
    if kind == "project":
        mark, ls = _cell_marks(p, seed)
        sim.set_field("mark", mark.cpu().numpy())
        sim.set_field("lsmerge", ls.cpu().numpy())
    s["fields"] = Fields(sim, PROJECT_FIELDS if kind == "project" else LEVELSET_FIELDS)
    return s


def run(state):
    kind, sim = state["kind"], state["sim"]
    if kind == "frames":
        if state["start"] is not None:
            sim.restore(state["start"])
        for _ in range(state["frames"]):
            sim.bubblesim()
        out = state["meshes"].take(sim)
        if state["start"] is not None:
            out["particles"] = state["particles"].take(sim)
        return out
    if kind == "project":
        sim.mapvelp2g_bubble()
        sim.setWaterBoundaryU(mp.TYPEAIR)
        sim.setWaterBoundaryU(mp.TYPEFLUID)
        sim.project_CG_bubble()
        return state["fields"].take(sim)
    if kind == "levelset":
        sim.computeLevelset(0.0)
        sim.sweepLSAndMardGrid()
        return state["fields"].take(sim)
    if kind == "surface":
        sim.hashAndSortParticles()
        sim.preMC()
        sim.runMC(mp.MC_FLUID)
        sim.runMC(mp.MC_GAS)
        return state["meshes"].take(sim)
    if state["v0"] is not None:
        loss = mp.dam_break_loss(state["v0"], sim, mp.PREC_MIXED)
        (grad,) = torch.autograd.grad(loss, state["v0"])
        return {"loss": loss.detach(), "grad": grad}
    loss, grad = sim.adj_gradient(None, mp.PREC_MIXED)
    return {"loss": loss, "grad": grad}


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
# floating-point operations of one particle-face, particle-node, particle-cell
# or particle-particle pair, counted from the formulas
PAIR_FLOPS = 20


def work(case):
    kind = case["kind"]
    n = (case["n"],) * 3 if "n" in case else (case["nx"], case["ny"], case["nz"])
    cells = n[0] * n[1] * n[2]
    liquid = {1: 0.6, 2: 0.4, 3: 0.5, 4: 0.24}.get(case.get("config"), LEVEL)
    parts = 8 * (n[0] - 2) * (n[1] - 2) * int(liquid * n[2])
    if kind == "frames":
        # particles (48 B) read and written, grid state of a step, and per
        # particle its pairs with 3 x 12 faces, 8 x 33 nodes of the 2x grid
        # and 4 neighbours
        k = case["frames"]
        return {"bytes": k * (96.0 * parts + 100.0 * cells), "flops": k * PAIR_FLOPS * 300.0 * parts}
    if kind == "project":
        return {"bytes": 32.0 * parts + (5 + 16.0) * cells, "flops": PAIR_FLOPS * 36.0 * parts + 400.0 * cells}
    if kind == "levelset":
        return {"bytes": 16.0 * parts + 13.0 * cells, "flops": PAIR_FLOPS * (1.0 * parts + 20 * cells)}
    if kind == "surface":
        # positions in, nodal fields of both surfaces formed, meshes out
        return {"bytes": 2 * 96.0 * parts + 2 * 32.0 * cells, "flops": PAIR_FLOPS * 264.0 * parts}
    k = case["steps"]
    return {"bytes": k * (96.0 * parts + 100.0 * cells), "flops": k * 2 * PAIR_FLOPS * 36.0 * parts}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind not in ("project", "levelset"):
        # whole simulated frames, surface meshes and gradients through frames
        # branch on rounded values throughout: they have no 64-bit value of
        # the same layout
        return None
    p = _column_params(case["nx"], case["ny"], case["nz"])
    pos, vel, flag = _column_particles(p, seed)
    if kind == "levelset":
        return _exact_levelset(p, pos, flag)
    return _exact_project(p, pos, vel, flag, *_cell_marks(p, seed))


def _cells_of(p, pos):
    """Cell coordinates of the particles, in the simulator's float32."""
    return [(pos[:, a] / np.float32(p.cellsize)).to(torch.int64) for a in range(3)]


def _faces64(p, pos, vel, axis, lo, hi, across, part):
    """Velocity component `axis` on its faces: kernel-weighted means over the
    cells lo..hi along the normal and -across..across in the other axes."""
    dims = [p.nx, p.ny, p.nz]
    dims[axis] += 1
    W = torch.zeros(dims[0] * dims[1] * dims[2], dtype=torch.float64, device="cuda")
    S = torch.zeros_like(W)
    pos, vel = pos[part], vel[part]
    cell = _cells_of(p, pos)
    rel = [pos[:, a].double() / p.cellsize for a in range(3)]
    m = float(p.m0)
    v = vel[:, axis].double()
    spans = [range(lo, hi + 1) if a == axis else range(-across, across + 1) for a in range(3)]
    for di in spans[0]:
        for dj in spans[1]:
            for dk in spans[2]:
                at = [cell[0] - di, cell[1] - dj, cell[2] - dk]
                ok = torch.ones_like(at[0], dtype=torch.bool)
                r2 = torch.zeros_like(v)
                for a in range(3):
                    ok &= (at[a] >= 0) & (at[a] < dims[a])
                    r2 += (rel[a] - at[a] - (0.0 if a == axis else 0.5)) ** 2
                w = m * torch.clamp(1.96 / torch.clamp(r2, min=1e-4) - 1.0, min=0.0)
                w = torch.where(ok, w, 0.0)
                idx = torch.where(ok, (at[0] * dims[1] + at[1]) * dims[2] + at[2], 0)
                W.index_add_(0, idx, w)
                S.index_add_(0, idx, w * v)
    return torch.where(W > 0, S / torch.where(W > 0, W, 1.0), 0.0).view(dims)


def _walls64(u):
    """setWaterBoundaryU with walls on the outer cell layer."""
    ux, uy, uz = u
    ux[:2], ux[-2:] = 0, 0
    uy[:, :2], uy[:, -2:] = 0, 0
    uz[:, :, -2] = torch.clamp(uz[:, :, -3], max=0.0) if uz.shape[2] > 5 else 0.0
    uz[:, :, :2], uz[:, :, -1] = 0, 0


def _shift(t, axis, d, fill):
    """t at the neighbour d along `axis`, `fill` outside."""
    out = torch.full_like(t, fill)
    n = t.shape[axis]
    out.narrow(axis, max(0, -d), n - 1).copy_(t.narrow(axis, max(0, d), n - 1))
    return out


def _exact_project(p, pos, vel, flag, mark, ls):
    h = float(p.cellsize)
    water, air = [], []
    for a in range(3):
        water.append(_faces64(p, pos, vel, a, -1, 0, 1, flag == mp.TYPEFLUID))
        air.append(_faces64(p, pos, vel, a, -2, 1, 2, flag == mp.TYPEAIR))
    del pos, vel, flag
    _walls64(air)
    _walls64(water)
    ls = ls.double()
    is_w, is_a = mark == mp.TYPEFLUID, mark == mp.TYPEAIR
    unknown = is_w | is_a
    div = torch.zeros_like(ls)
    for a in range(3):
        n = ls.shape[a]
        for d in (1, -1):
            wv, av = (u[a].narrow(a, 1 if d > 0 else 0, n) for u in (water, air))
            nw, na = _shift(is_w, a, d, False), _shift(is_a, a, d, False)
            ln = _shift(ls, a, d, 0.0)
            mixed = (is_w & na) | (is_a & nw)
            th = torch.where(mixed, -ls / torch.where(mixed, ln - ls, 1.0), 1.0)
            own, other = torch.where(is_w, wv, av), torch.where(is_w, av, wv)
            div += d * (th * own + (1 - th) * other)
    b = torch.where(unknown, div / h, 0.0)
    del div, air
    # neighbours that are walls take the centre's value
    wall = mark == mp.TYPEBOUNDARY
    diag = -6.0 + sum(_shift(wall, a, d, True).double() for a in range(3) for d in (1, -1))
    del wall

    def apply(x):
        s = diag * x
        for a in range(3):
            n = x.shape[a]
            s.narrow(a, 0, n - 1).add_(x.narrow(a, 1, n - 1))
            s.narrow(a, 1, n - 1).add_(x.narrow(a, 0, n - 1))
        return torch.where(unknown, s / (h * h), 0.0)

    x = torch.zeros_like(b)
    r = b.clone()
    q = r.clone()
    rr = float((r * r).sum())
    stop = rr * 1e-22
    for _ in range(6000):
        if rr <= stop:
            break
        z = apply(q)
        alpha = rr / float((q * z).sum())
        x.add_(q, alpha=alpha)
        r.add_(z, alpha=-alpha)
        new = float((r * r).sum())
        q.mul_(new / rr).add_(r)
        rr = new
    for a in range(3):
        n = x.shape[a]
        water[a].narrow(a, 1, n - 1).sub_((x.narrow(a, 1, n - 1) - x.narrow(a, 0, n - 1)) / h)
    return {"press": x.reshape(-1), "waterux": water[0].reshape(-1), "wateruy": water[1].reshape(-1),
            "wateruz": water[2].reshape(-1)}


def _nearest64(p, pos, part):
    """Distance from each cell centre to the nearest particle in the 5^3 cells
    around it, at most 2.5 cells, less half a cell."""
    dims, h = (p.nx, p.ny, p.nz), float(p.cellsize)
    best = torch.full((dims[0] * dims[1] * dims[2],), (2.5 * h) ** 2, dtype=torch.float64, device="cuda")
    pos = pos[part]
    cell = _cells_of(p, pos)
    x = [pos[:, a].double() for a in range(3)]
    for di in range(-2, 3):
        for dj in range(-2, 3):
            for dk in range(-2, 3):
                at = [cell[0] - di, cell[1] - dj, cell[2] - dk]
                ok = torch.ones_like(at[0], dtype=torch.bool)
                d2 = torch.zeros_like(x[0])
                for a in range(3):
                    ok &= (at[a] >= 0) & (at[a] < dims[a])
                    d2 += (x[a] - (at[a] + 0.5) * h) ** 2
                idx = torch.where(ok, (at[0] * dims[1] + at[1]) * dims[2] + at[2], 0)
                best.scatter_reduce_(0, idx, torch.where(ok, d2, 1e30), "amin")
    return (torch.sqrt(best) - 0.5 * h).view(dims)


def _sweeps64(v, held, passes=5):
    """Jacobi passes of the distance update over the eight octants."""
    for _ in range(passes):
        res = v.clone()
        near = {(a, d): _shift(v, a, d, float("inf")) for a in range(3) for d in (-1, 1)}
        for di in (-1, 1):
            for dj in (-1, 1):
                for dk in (-1, 1):
                    a, b, c = near[0, di], near[1, dj], near[2, dk]
                    inside = torch.isfinite(a) & torch.isfinite(b) & torch.isfinite(c)
                    a, b, c = (torch.where(inside, t, 0.0) for t in (a, b, c))
                    d = torch.minimum(a, torch.minimum(b, c)) + 1
                    far = d > torch.maximum(a, torch.maximum(b, c))
                    disc = torch.clamp(3 - (a - b) ** 2 - (a - c) ** 2 - (b - c) ** 2, min=0.0)
                    d = torch.where(far, (a + b + c + torch.sqrt(disc)) / 3, d)
                    res = torch.where(inside & ~held & (d < res), d, res)
        v = res
    return v


def _exact_levelset(p, pos, flag):
    h = float(p.cellsize)
    ls = []
    for t in (mp.TYPEFLUID, mp.TYPEAIR):
        v = _nearest64(p, pos, flag == t) / h
        far = v > 1.99
        v = _sweeps64(torch.where(far, 5.0, v), ~far)
        v = -v
        far = v > 0
        v = _sweeps64(torch.where(far, 5.0, v), ~far)
        ls.append(-v * h)
    lf, la = ls
    merged = torch.where(la > 4.99 * h, lf, torch.where(lf > 4.99 * h, la, torch.where(
        (la > 0.8 * h) & (lf > 0.8 * h), torch.minimum(lf, la), (lf - la) * 0.5)))
    for a in range(3):
        merged.select(a, 0).fill_(-0.5 * h)
        merged.select(a, merged.shape[a] - 1).fill_(-0.5 * h)
    return {"lsmerge": merged.reshape(-1), "lsfluid": lf.reshape(-1), "lsair": la.reshape(-1), "mark": None}
