"""What the engine is timed on: the calls a program that uses it makes.

  step     one PBFluids step (all substeps and solver iterations) of one scene whose state the program holds on the
           GPU: uploaded, stepped, read back.  From a few thousand particles, where launches and latency are all
           there is, to the 4M-particle dam break.
  batch    one step of many independent scenes of uneven sizes (pbf_b200.Batch).
  adjoint  one differentiable step, forward and backward, through torch.autograd.
  mesh     a deformed triangle mesh refitted: LBVH, signed-distance grid, closest-point queries.
  coupled  one frame of the two-way coupled loop: fluid step, contact forces, host deformation, mesh refit.

Scene sizes and constants are those of pbf_b200.scenes, pbf_b200.presets and bench.py.  Particles start as a block
in motion: the lattice of the scene with every particle displaced by up to a fifth of the spacing per axis and given
a random velocity, as a fluid has it after its first steps.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "realtime-fsi-engine_b200"))

import pbf_b200 as P  # noqa: E402
from pbf_b200 import adjoint as A  # noqa: E402
from pbf_b200 import fsi, presets  # noqa: E402
from pbf_b200 import scenes as S  # noqa: E402

DEV = "cuda:0"


# ---- the cases ----------------------------------------------------------------------------------------------------
def _step(name, nx, ny, nz, d=0.02, box=(1.6, 1.0, 1.0), substeps=2, iterations=4, dt=1.0 / 60.0, scorr=True,
          vorticity=True, obstacle="none", graph=False, preset=-1):
    return dict(name=name, kind="step", nx=nx, ny=ny, nz=nz, d=d, bx=box[0], by=box[1], bz=box[2], substeps=substeps,
                iterations=iterations, dt=dt, scorr=scorr, vorticity=vorticity, obstacle=obstacle, graph=graph,
                preset=preset)


def listed():
    return [
        # the smallest scene anyone steps (a first try, a unit test): launches and latency
        _step("step-2k", 13, 13, 13),
        # the reference application's "Surface Cube" preset: 16,384 particles over a mesh, launched pass by pass
        _step("step-preset-16k", 0, 0, 0, obstacle="mesh", preset=1),
        # the small dam break, replayed from its CUDA graph in a real-time loop
        _step("step-32k", 32, 32, 32, graph=True),
        # the coupled scene's fluid alone: a quarter of a million particles over a mesh
        _step("step-262k", 64, 64, 64, d=0.0125, box=(1.6, 1.6, 1.0), obstacle="mesh", graph=True),
        # a ragged block in between, an incompressible solve without the tensile and vorticity terms
        _step("step-0.6M", 101, 89, 67, d=0.01, box=(2.0, 1.2, 1.0), substeps=1, dt=1.0 / 120.0, scorr=False,
              vorticity=False, obstacle="sphere"),
        # the large dam break (bench.py's workload)
        _step("step-4M", 256, 128, 128, d=0.005, box=(2.0, 1.0, 1.0), substeps=1, dt=1.0 / 120.0, obstacle="capsule",
              graph=True),
        # a few small scenes at once, as a parameter sweep runs them
        dict(name="batch-12", kind="batch", scenes=12, lo=700, hi=12000, sizes=3),
        # the 64-scene batch of bench.py
        dict(name="batch-64", kind="batch", scenes=64, lo=4096, hi=131072, sizes=7),
        # the differentiable dam break: one scene, and sixteen in one batch (the smooth variant, whose gradient is
        # usable: s_corr off, cohesion 0)
        dict(name="adjoint-1", kind="adjoint", scenes=1, side=32, substeps=16),
        dict(name="adjoint-16", kind="adjoint", scenes=16, side=32, substeps=16),
        # the deforming sphere's collision field, as the coupled loop refreshes it, with queries against it
        dict(name="mesh-5k", kind="mesh", subdiv=4, cell=0.0125, queries=20000, rebuild=False),
        # the coupled frame itself
        dict(name="coupled-262k", kind="coupled", side=64, subdiv=4),
    ]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "batch", "adjoint", "mesh", "coupled"])

    def spread(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    if kind == "step":
        n = spread(1000, 4000000)
        a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
        side = n ** (1.0 / 3.0)
        ny, nz = max(5, int(side * a)), max(5, int(side * b))
        nx = max(5, int(n / (ny * nz)))
        # the box holds the block with room to fall into; the hash table follows the particle count
        d = 0.02 if n < 6e4 else 0.0125 if n < 4e5 else 0.005
        box = tuple(round(max(0.5, m * d * rng.uniform(1.1, 2.0)), 3) for m in (nx, ny, nz))
        substeps = 2 if n < 4e5 else 1
        case = _step("", nx, ny, nz, d, box, substeps, rng.choice([3, 4, 4, 5]), substeps / 120.0,
                     rng.random() < 0.7, rng.random() < 0.7, rng.choice(["none", "sphere", "mesh"]),
                     rng.random() < 0.5)
        del case["name"]
        return case
    if kind == "batch":
        lo = int(spread(500, 10000))
        return dict(kind="batch", scenes=rng.randint(2, 48), lo=lo, hi=int(lo * rng.uniform(2, 12)),
                    sizes=rng.randint(0, 10 ** 6))
    if kind == "adjoint":
        return dict(kind="adjoint", scenes=rng.randint(1, 12), side=rng.randint(12, 32), substeps=rng.randint(2, 12))
    if kind == "mesh":
        return dict(kind="mesh", subdiv=rng.randint(2, 5), cell=round(spread(0.008, 0.03), 4),
                    queries=int(spread(100, 50000)), rebuild=rng.random() < 0.5)
    return dict(kind="coupled", side=rng.randint(20, 64), subdiv=rng.randint(3, 4))


# ---- inputs -------------------------------------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _moving(base, d, dt, lo, hi, seed):
    """(pos, vel) as float4 tensors: `base` displaced by up to 0.2 d per axis (kept inside the walls), random
    velocities of a tenth of a spacing per substep."""
    g = _gen(seed)
    pos = torch.as_tensor(base, dtype=torch.float32, device=DEV)
    n = len(pos)
    pos = pos + (torch.rand((n, 3), generator=g, device=DEV) * 2 - 1) * (0.2 * d)
    lo, hi = (torch.tensor(list(v), dtype=torch.float32, device=DEV) for v in (lo, hi))
    pos = torch.minimum(torch.maximum(pos, lo + 1e-3 * d), hi - 1e-3 * d)
    vel = torch.randn((n, 3), generator=g, device=DEV) * (0.1 * d / dt)
    p4, v4 = torch.zeros((n, 4), device=DEV), torch.zeros((n, 4), device=DEV)
    p4[:, :3], v4[:, :3] = pos, vel
    return p4, v4


def _scene(case):
    """(cfg, lattice, obstacle) of a step case; the obstacle is None, ("grid", dist, origin, cell, padding) or
    ("mesh", verts, faces, cell, padding)."""
    if case["preset"] >= 0:
        pre = presets.presets()[case["preset"]]
        cfg = pre.fluid
        base = presets.spawn_particles(cfg)["pos"].copy()
        v, f = S.icosphere(3, 1.0, (0.0, 0.0, 0.0))
        v = presets.fit_mesh(v, presets.fit_center(cfg), pre.mesh_fit_size)
        v = presets.place_mesh(v, pre.mesh_translate[:], pre.mesh_rot_deg[:])
        return cfg, base, ("mesh", v, f, pre.sdf_cell, pre.sdf_padding)
    d = case["d"]
    n = case["nx"] * case["ny"] * case["nz"]
    box = (case["bx"], case["by"], case["bz"])
    cfg = S.base_config(2 * d, d, box, case["substeps"], case["iterations"], case["dt"], n)
    cfg.enable_scorr = int(case["scorr"])
    cfg.enable_vorticity = int(case["vorticity"])
    base = S.lattice(case["nx"], case["ny"], case["nz"], d, (0.0, 0.0, 0.0), 0.0, 0)
    # an obstacle at the far end of the block
    reach = case["nx"] * d
    centre = (min(reach + 0.1, box[0]), 0.3 * box[1], 0.5 * box[2])
    if case["obstacle"] == "capsule":
        grid, origin, cell = S.capsule_grid(S.C2_CAPSULE["radius"], S.C2_CAPSULE["a"], S.C2_CAPSULE["b"], d)
        return cfg, base, ("grid", grid, origin, cell, d / 2)
    if case["obstacle"] == "sphere":
        grid, origin, cell = S.sphere_grid(0.15, centre, max(d, 0.01))
        return cfg, base, ("grid", grid, origin, cell, d / 2)
    if case["obstacle"] == "mesh":
        v, f = S.icosphere(4, 0.2, centre)
        return cfg, base, ("mesh", v, f, 0.0125, 0.0125 / 2)
    return cfg, base, None


def _upload(fl, p4, v4):
    P._capi.check(P.lib().pbf_set_particles_device(fl.handle, p4.data_ptr(), v4.data_ptr(), len(p4)))


def _download(fl, p4, v4):
    P._capi.check(P.lib().pbf_read_particles_device(fl.handle, p4.data_ptr(), v4.data_ptr(), len(p4)))


def _prepare_step(case, seed):
    cfg, base, obstacle = _scene(case)
    dt = cfg.dt / cfg.substep_iterations
    p4, v4 = _moving(base, cfg.spacing, dt, cfg.bounds_min, cfg.bounds_max, seed)
    fl = P.PBFluids(cfg)
    st = dict(kind="step", fluid=fl, pos=p4, vel=v4, out=(torch.empty_like(p4), torch.empty_like(v4)), cfg=cfg)
    if obstacle is not None:
        if obstacle[0] == "grid":
            st["sdf"] = P.GridSDF(obstacle[1], obstacle[2], obstacle[3])
        else:
            st["sdf"] = P.SDFBoundary()
            st["sdf"].buildFromMesh(obstacle[1], obstacle[2], obstacle[3])
        fl.setSDFBoundary(st["sdf"])
        fl.setSDFPadding(obstacle[4])
    torch.cuda.synchronize()
    if case["graph"]:
        fl.set_use_graph(True)
    _upload(fl, p4, v4)
    fl.step()  # buffers and, with it on, the graph
    fl.sync()
    return st


def _batch_scenes(case):
    sizes = np.exp(np.random.default_rng(case["sizes"]).uniform(math.log(case["lo"]), math.log(case["hi"]),
                                                                case["scenes"])).astype(int)
    return S.c3(case["sizes"], case["scenes"], sizes)


def _prepare_batch(case, seed):
    cfg, scenes = _batch_scenes(case)
    b = P.Batch(cfg, scenes)
    ps, vs = [], []
    for k, s in enumerate(scenes):
        grid, origin, cell, pad = s["sdf"]
        b.set_sdf_grid(k, grid, origin, cell)
        b.set_sdf_mode(k, pad, False)
        p4, v4 = _moving(s["pos"], cfg.spacing, cfg.dt / cfg.substep_iterations, s["bounds_min"], s["bounds_max"],
                         seed * 1000 + k)
        ps.append(p4)
        vs.append(v4)
    p4, v4 = torch.cat(ps), torch.cat(vs)
    torch.cuda.synchronize()
    b.set_state(p4.data_ptr(), v4.data_ptr())
    b.step()
    b.sync()
    return dict(kind="batch", batch=b, pos=p4, vel=v4, out=(torch.empty_like(p4), torch.empty_like(v4)))


_SPHERE = (0.15, (0.78, 0.32, 0.32))


def _adjoint_inputs(case, seed):
    d, side, k = 0.02, case["side"], case["scenes"]
    n = side ** 3
    cfg = S.base_config(2 * d, d, (1.6, 1.0, 1.0), case["substeps"], 4, 1.0 / 60.0, n, 1 << 17)
    cfg.enable_scorr = 0
    cfg.cohesion_strength = 0.0
    base = S.lattice(side, side, side, d, (0.0, 0.0, 0.0), 0.0, 0)
    g = _gen(seed)
    pos = torch.as_tensor(base, device=DEV).repeat(k, 1)
    pos = pos + (torch.rand((k * n, 3), generator=g, device=DEV) * 2 - 1) * 0.001
    vel = torch.randn((k * n, 3), generator=g, device=DEV) * 0.02
    shift = torch.tensor([0.3, 0.0, 0.1], device=DEV)
    target = pos + shift + torch.randn((k * n, 3), generator=g, device=DEV) * 0.01
    return cfg, n, pos.contiguous(), vel, target


def _prepare_adjoint(case, seed):
    cfg, n, pos, vel, target = _adjoint_inputs(case, seed)
    sc = [dict(n=n, bounds_min=tuple(cfg.bounds_min), bounds_max=tuple(cfg.bounds_max), hash_size=cfg.hash_size)
          for _ in range(case["scenes"])]
    b = P.Batch(cfg, sc)
    grid, origin, cell = S.sphere_grid(_SPHERE[0], _SPHERE[1], 0.02)
    for k in range(case["scenes"]):
        b.set_sdf_grid(k, grid, origin, cell)
        b.set_sdf_mode(k, 0.01, False)
    st = dict(kind="adjoint", batch=b, pos=pos.requires_grad_(), vel=vel.requires_grad_(), target=target,
              offset=torch.zeros((case["scenes"], 3), requires_grad=True))
    _run_adjoint(st)  # buffers and graphs
    return st


def _deformed(subdiv, seed):
    """The sphere of the coupled scene pushed in and out by a few smooth waves and fitted to one box, so that the
    grid of a rebuild has the same size whatever the seed."""
    v, f = S.icosphere(subdiv, 0.2, (0.0, 0.0, 0.0))
    rng = np.random.default_rng(seed)
    bump = np.zeros(len(v))
    for _ in range(4):
        k = rng.normal(size=3) * 15.0
        bump += rng.uniform(0.002, 0.008) * np.sin(v @ k + rng.uniform(0, 6.28))
    c = np.array([0.8, 0.3, 0.5])
    moved = v * (1.0 + bump[:, None] / 0.2)
    lo, hi = moved.min(0), moved.max(0)
    return v + c, f, (moved - (lo + hi) / 2) * (0.4 * 0.9903 / (hi - lo)) + c


def _prepare_mesh(case, seed):
    rest, f, moved = _deformed(case["subdiv"], seed)
    pts = np.random.default_rng(seed + 1).uniform([0.5, 0.0, 0.2], [1.1, 0.6, 0.8], (case["queries"], 3))
    sdf = P.SDFBoundary()
    sdf.buildFromMesh(rest, f, case["cell"])
    return dict(kind="mesh", sdf=sdf, verts=moved, faces=f, pts=pts.astype(np.float32), cell=case["cell"],
                rebuild=case["rebuild"])


def _prepare_coupled(case, seed):
    # the coupled scene's block, lowered until its underside surrounds the top of the sphere
    d, side = 0.0125, case["side"]
    box = (1.6, 1.6, 1.0)
    v, f = S.icosphere(case["subdiv"], 0.2, (0.8, 0.3, 0.5))
    base = S.lattice(side, side + 8, side, d, (0.8 - side * d / 2, 0.42, 0.5 - side * d / 2), 0.0, 0)
    out = np.linalg.norm(base - np.array([0.8, 0.3, 0.5], np.float32), axis=1) > 0.2 + d
    base = base[out][: side ** 3]
    cfg = S.base_config(2 * d, d, box, 2, 4, 1.0 / 60.0, len(base))
    p4, v4 = _moving(base, d, 1.0 / 120.0, cfg.bounds_min, cfg.bounds_max, seed)
    v4[:, 1] -= 1.0
    prm, kring, band = fsi.c1_deform_params()
    host = p4[:, :3].cpu().numpy()
    sc = fsi.CoupledScene(cfg, host, np.zeros_like(host), v, f, np.argsort(v[:, 1], kind="stable")[:16], d, prm, band,
                          kring=kring, incremental=True)
    st = dict(kind="coupled", scene=sc, pos=p4, vel=v4, out=(torch.empty_like(p4), torch.empty_like(v4)))
    torch.cuda.synchronize()
    _run_coupled(st)
    return st


def prepare(case, seed):
    return {"step": _prepare_step, "batch": _prepare_batch, "adjoint": _prepare_adjoint, "mesh": _prepare_mesh,
            "coupled": _prepare_coupled}[case["kind"]](case, seed)


# ---- one pass -----------------------------------------------------------------------------------------------------
def _run_step(st):
    fl = st["fluid"]
    _upload(fl, st["pos"], st["vel"])
    fl.step()
    _download(fl, *st["out"])
    fl.sync()  # the solver has a stream of its own: what reads the tensors next is not ordered behind it
    return {"pos": st["out"][0], "vel": st["out"][1]}


def _run_batch(st):
    b = st["batch"]
    b.set_state(st["pos"].data_ptr(), st["vel"].data_ptr())
    b.step()
    b.get_state(st["out"][0].data_ptr(), st["out"][1].data_ptr())
    return {"pos": st["out"][0], "vel": st["out"][1]}


def _run_adjoint(st):
    pos, vel, off = st["pos"], st["vel"], st["offset"]
    pos.grad = vel.grad = off.grad = None
    p, v = A.step(st["batch"], pos, vel, off)
    ((p - st["target"]) ** 2).sum(1).mean().backward()
    return {"pos": p, "vel": v, "gpos": pos.grad, "gvel": vel.grad, "goffset": off.grad}


def _run_mesh(st):
    if st["rebuild"]:
        st["sdf"].buildFromMesh(st["verts"], st["faces"], st["cell"])
    else:
        st["sdf"].refitFromMesh(st["verts"])
    dist = st["sdf"].distances()
    face, point = st["sdf"].closest_many(st["pts"])
    return {"dist": dist, "face": face, "point": point}


def _run_coupled(st):
    sc = st["scene"]
    _upload(sc.fluid, st["pos"], st["vel"])
    forces, _ = sc.frame()
    _download(sc.fluid, *st["out"])
    sc.fluid.sync()
    return {"pos": st["out"][0], "vel": st["out"][1], "forces": forces, "verts": sc.deform.vertices()}


def run(state):
    return {"step": _run_step, "batch": _run_batch, "adjoint": _run_adjoint, "mesh": _run_mesh,
            "coupled": _run_coupled}[state["kind"]](state)


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
PAIRS = 30  # in-range neighbours of a particle of a resting fluid at h = 2 d


def _substep_flops(iterations, vorticity):
    # per pair: lambda 27 (distance 8, poly6 4, gradient 9, sums 6), delta-p 19, integrate 20, vorticity 18
    return PAIRS * (iterations * (27 + 19) + 20 + (18 if vorticity else 0))


def work(case):
    kind = case["kind"]
    if kind == "step":
        n, sub, it, vort = case["nx"] * case["ny"] * case["nz"], case["substeps"], case["iterations"], case["vorticity"]
        if case["preset"] >= 0:
            c = presets.presets()[case["preset"]].fluid
            n, sub, it, vort = c.particle_count, c.substep_iterations, c.solver_iterations, bool(c.enable_vorticity)
        return {"bytes": 64.0 * n, "flops": float(n) * sub * _substep_flops(it, vort)}
    if kind == "batch":
        n = sum(s["n"] for s in _batch_scenes(case)[1])
        return {"bytes": 64.0 * n, "flops": n * 2.0 * _substep_flops(4, True)}
    if kind == "adjoint":
        # the forward, its recomputation and a reverse pass of about twice its arithmetic; state and gradients
        n = case["scenes"] * case["side"] ** 3
        return {"bytes": 96.0 * n, "flops": 4.0 * n * case["substeps"] * _substep_flops(4, False)}
    if kind == "mesh":
        # vertices in, the grid and the queries' answers out; the log of the face count boxes and one face each
        nf, vox = 20 * 4 ** case["subdiv"], (math.ceil(0.4 / case["cell"]) + 10) ** 3
        q = vox + case["queries"]
        return {"bytes": 12.0 * nf + 4.0 * vox + 28.0 * case["queries"], "flops": q * (12.0 * math.log2(nf) + 60.0)}
    n = case["side"] ** 3
    return {"bytes": 64.0 * n, "flops": float(n) * 2 * _substep_flops(4, True)}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------
def _hash(c, mask):
    m = 0xFFFFFFFF
    return ((c[:, 0] * 73856093 & m) ^ (c[:, 1] * 19349663 & m) ^ (c[:, 2] * 83492791 & m)) & mask


class _Buckets:
    """The reference's neighbour candidates: particles by the hash of their predicted cell, a query reading the 27
    buckets around its current cell (one that collides as often as it is met)."""

    def __init__(self, x, h, hash_size):
        self.h, self.mask = h, hash_size - 1
        key = _hash(torch.floor(x.detach() / h).long(), self.mask)
        self.key, self.ids = torch.sort(key, stable=True)

    def pairs(self, x):
        x = x.detach()
        cell = torch.floor(x / self.h).long()
        out_i, out_j = [], []
        ar = torch.arange(len(x), device=x.device)
        for k in range(27):
            off = torch.tensor([k % 3 - 1, k // 3 % 3 - 1, k // 9 - 1], device=x.device)
            q = _hash(cell + off, self.mask)
            lo = torch.searchsorted(self.key, q)
            cnt = torch.searchsorted(self.key, q, right=True) - lo
            i = torch.repeat_interleave(ar, cnt)
            first = torch.cumsum(cnt, 0) - cnt
            j = self.ids[lo[i] + torch.arange(len(i), device=x.device) - first[i]]
            near = ((x[i] - x[j]) ** 2).sum(1) <= self.h * self.h
            near &= i != j
            out_i.append(i[near])
            out_j.append(j[near])
        return torch.cat(out_i), torch.cat(out_j)


def _sample(grid, p):
    dist, origin, cell = grid
    top = torch.tensor([s - 1.0 for s in dist.shape], dtype=p.dtype, device=p.device)
    u = torch.minimum(torch.clamp((p - origin) / cell, min=0.0), top)
    b = torch.floor(u.detach())
    f = u - b
    b = b.long()
    e = torch.minimum(b + 1, top.long())
    out = 0.0
    for k in range(8):
        ix = [(e if k >> a & 1 else b)[:, a] for a in range(3)]
        w = 1.0
        for a in range(3):
            w = w * (f[:, a] if k >> a & 1 else 1.0 - f[:, a])
        out = out + w * dist[ix[0], ix[1], ix[2]]
    return out


def _project(grid, pad, p):
    """The push out of the obstacle: (moved p, contact, normal)."""
    d = _sample(grid, p)
    e = torch.eye(3, dtype=p.dtype, device=p.device) * grid[2]
    g = torch.stack([(_sample(grid, p + e[a]) - _sample(grid, p - e[a])) / (2 * grid[2]) for a in range(3)], 1)
    g2 = (g * g).sum(1)
    hit = (d < pad) & (g2 > 1e-12)
    n = g / torch.sqrt(torch.where(hit, g2, torch.ones_like(g2)))[:, None]
    return torch.where(hit[:, None], p + n * (pad - d)[:, None], p), hit, n


class _Solver64:
    def __init__(self, cfg, grid=None, pad=0.0):
        self.c, self.grid, self.pad = cfg, grid, pad
        t = dict(dtype=torch.float64, device=DEV)
        self.h, self.dt = float(cfg.h), float(np.float32(cfg.dt) / np.float32(cfg.substep_iterations))
        self.lo = torch.tensor(list(cfg.bounds_min), **t)
        self.hi = torch.tensor(list(cfg.bounds_max), **t)
        self.g = torch.tensor(list(cfg.gravity), **t)
        self.k6 = 315.0 / (64.0 * math.pi * self.h ** 9)
        self.ks = 45.0 / (math.pi * self.h ** 6)

    def _geom(self, x, i, j):
        r = x[i] - x[j]
        r2 = (r * r).sum(1)
        w = self.k6 * (self.h ** 2 - r2) ** 3
        some = r2 >= 1e-10
        q = torch.sqrt(torch.where(some, r2, torch.ones_like(r2)))
        s = torch.where(some, -self.ks * (self.h - q) ** 2 / q, torch.zeros_like(q))
        return w, r * s[:, None]

    def _sum(self, n, i, v):
        return torch.zeros((n,) + v.shape[1:], dtype=v.dtype, device=v.device).index_add(0, i, v)

    def substep(self, p0, v0, grid=None):
        """(pos, vel, omega, buckets) after one substep."""
        c, n, grid = self.c, len(p0), grid or self.grid
        v1 = v0 + self.g * self.dt
        x = p0 + v1 * self.dt
        buckets = _Buckets(x, self.h, c.hash_size)
        wq = self.k6 * (self.h ** 2 - (c.delta_q * self.h) ** 2) ** 3
        for _ in range(c.solver_iterations):
            i, j = buckets.pairs(x)
            w, a = self._geom(x, i, j)
            rho = self.k6 * self.h ** 6 + self._sum(n, i, w)
            grad = self._sum(n, i, a) / c.rho0
            den = self._sum(n, i, (a * a).sum(1)) / c.rho0 ** 2 + (grad * grad).sum(1) + c.eps
            lam = -torch.clamp(rho / c.rho0 - 1.0, min=-c.cohesion_strength) / den
            f = lam[i] + lam[j]
            if c.enable_scorr:
                f = f - c.k_corr * (w / wq) ** c.n_corr
            dp = self._sum(n, i, f[:, None] * a) / c.rho0
            l2, top = (dp * dp).sum(1), 0.5 * self.h
            far = l2 > top * top
            dp = torch.where(far[:, None], dp * (top / torch.sqrt(torch.where(far, l2, torch.ones_like(l2))))[:, None],
                             dp)
            x = x + dp
            if grid is not None:
                x = _project(grid, self.pad, x)[0]
        push, omega = 0.0, None
        if c.enable_viscosity or c.enable_vorticity:
            i, j = buckets.pairs(x)
            w, a = self._geom(x, i, j)
            u = v1[j] - v1[i]
            if c.enable_viscosity:
                push = self._sum(n, i, u * w[:, None]) / c.rho0 * c.viscosity
            if c.enable_vorticity:
                omega = self._sum(n, i, torch.linalg.cross(u, a)) / c.rho0
        low, high = x <= self.lo, x >= self.hi
        x = torch.where(low, self.lo, torch.where(high, self.hi, x))
        if grid is not None:
            x, hit, nrm = _project(grid, self.pad, x)
        v = (x - p0) / self.dt + push
        s2 = (v * v).sum(1)
        fast = s2 > 2500.0
        v = torch.where(fast[:, None], v * (50.0 / torch.sqrt(torch.where(fast, s2, torch.ones_like(s2))))[:, None], v)
        v = torch.where(low | high, v * -c.bound_damping, v)
        if grid is not None:
            v = torch.where(hit[:, None], v - nrm * (v * nrm).sum(1, keepdim=True), v)
        return x, v, omega, buckets

    def confine(self, x, v, omega, buckets):
        if omega is None:
            return v
        i, j = buckets.pairs(x)
        _, a = self._geom(x, i, j)
        # a smooth |omega| where omega vanishes, so that its gradient is zero there
        m2 = (omega * omega).sum(1)
        mag = torch.where(m2 > 0, torch.sqrt(torch.where(m2 > 0, m2, torch.ones_like(m2))), torch.zeros_like(m2))
        eta = self._sum(len(x), i, a * mag[j][:, None]) / self.c.rho0
        e2 = (eta * eta).sum(1)
        on = e2 >= 1e-12
        nn = eta / torch.sqrt(torch.where(on, e2, torch.ones_like(e2)))[:, None]
        dv = self.c.vorticity_epsilon * torch.linalg.cross(nn, omega) * self.dt
        return torch.where(on[:, None], v + dv, v)

    def step(self, p, v):
        for _ in range(self.c.substep_iterations):
            p, v, omega, buckets = self.substep(p, v)
        return p, self.confine(p, v, omega, buckets)

    def gradients(self, p, v, loss):
        """d loss(final p) / d (p, v, translation of the obstacle), substep by substep in reverse."""
        saved = []
        with torch.no_grad():
            q, u = p, v
            for _ in range(self.c.substep_iterations):
                saved.append((q, u))
                q, u, omega, buckets = self.substep(q, u)
        out = (q, self.confine(q, u, omega, buckets))
        end = q.clone().requires_grad_()
        gp, = torch.autograd.grad(loss(end), end)
        gv = torch.zeros_like(gp)
        gt = torch.zeros(3, dtype=torch.float64, device=DEV)
        for q, u in reversed(saved):
            q, u = q.clone().requires_grad_(), u.clone().requires_grad_()
            t = torch.zeros(3, dtype=torch.float64, device=DEV, requires_grad=True)
            grid = (self.grid[0], self.grid[1] + t, self.grid[2])
            x, w, _, _ = self.substep(q, u, grid)
            gp, gv, ti = torch.autograd.grad((x, w), (q, u, t), (gp, gv), allow_unused=True)
            gt = gt + (ti if ti is not None else 0.0)
        return out, gp, gv, gt


def _grid64(dist, origin, cell):
    return (torch.as_tensor(np.asarray(dist, np.float32), device=DEV).double(),
            torch.tensor([float(np.float32(o)) for o in origin], dtype=torch.float64, device=DEV),
            float(np.float32(cell)))


def _pad4(x):
    return torch.cat([x, torch.zeros((len(x), 1), dtype=x.dtype, device=x.device)], 1)


def _closest64(tri, p):
    """Distance, closest point and winding number of points against every triangle."""
    a, b, c = (tri[None, :, k] for k in range(3))
    p = p[:, None]
    ab, ac, bc = b - a, c - a, c - b

    def dot(x, y):
        return (x * y).sum(-1, keepdim=True)

    def on(start, edge):
        return start + edge * torch.clamp(dot(p - start, edge) / dot(edge, edge), 0.0, 1.0)

    nrm = torch.linalg.cross(ab, ac)
    flat = p - nrm * (dot(p - a, nrm) / dot(nrm, nrm))
    inside = ((dot(torch.linalg.cross(ab, flat - a), nrm) >= 0) & (dot(torch.linalg.cross(bc, flat - b), nrm) >= 0)
              & (dot(torch.linalg.cross(-ac, flat - c), nrm) >= 0))
    best, point = None, None
    for q in (on(a, ab), on(a, ac), on(b, bc), flat):
        d = dot(p - q, p - q)
        if q is flat:
            d = torch.where(inside, d, torch.full_like(d, math.inf))
        if best is None:
            best, point = d, q.expand(d.shape[:-1] + (3,))
        else:
            point = torch.where(d < best, q, point)
            best = torch.minimum(best, d)
    d, k = best[..., 0].min(1)
    u, v, w = (x / torch.sqrt(dot(x, x)).clamp_min(1e-300) for x in (a - p, b - p, c - p))
    turn = 2.0 * torch.atan2((u * torch.linalg.cross(v, w)).sum(-1),
                             1.0 + (u * v).sum(-1) + (v * w).sum(-1) + (w * u).sum(-1)).sum(1)
    return torch.sqrt(d), point[torch.arange(len(k), device=k.device), k], turn / (4 * math.pi)


def _mesh64(verts, faces, pts):
    tri = torch.as_tensor(np.asarray(verts), device=DEV).double()[torch.as_tensor(np.asarray(faces), device=DEV).long()]
    pts = torch.as_tensor(np.asarray(pts), device=DEV).double()
    step = max(1, 6000000 // len(tri))
    got = [_closest64(tri, pts[k:k + step]) for k in range(0, len(pts), step)]
    return [torch.cat([g[m] for g in got]) for m in range(3)]


def exact(case, seed):
    """With the scenes' tensile term (k = 0.1 at unit mass) the solver magnifies a rounding about five times per
    iteration, so that after two substeps 32-bit and 64-bit velocities have parted: those steps have no value here
    (the presets' term, a hundred times weaker, has)."""
    kind = case["kind"]
    tame = kind == "step" and (case["preset"] >= 0 or not case["scorr"])
    if tame and case["nx"] * case["ny"] * case["nz"] < 700000:
        cfg, base, obstacle = _scene(case)
        p4, v4 = _moving(base, cfg.spacing, cfg.dt / cfg.substep_iterations, cfg.bounds_min, cfg.bounds_max, seed)
        grid, pad = None, 0.0
        if obstacle is not None and obstacle[0] == "grid":
            grid, pad = _grid64(*obstacle[1:4]), obstacle[4]
        elif obstacle is not None:
            dist, origin = _mesh_grid64(obstacle[1], obstacle[2], obstacle[3])
            grid, pad = _grid64(dist, origin, obstacle[3]), obstacle[4]
        with torch.no_grad():
            p, v = _Solver64(cfg, grid, float(np.float32(pad))).step(p4[:, :3].double(), v4[:, :3].double())
        return {"pos": _pad4(p), "vel": _pad4(v)}
    if kind == "adjoint" and case["scenes"] * case["side"] ** 3 < 70000:
        cfg, n, pos, vel, target = _adjoint_inputs(case, seed)
        grid, origin, cell = S.sphere_grid(_SPHERE[0], _SPHERE[1], 0.02)
        sol = _Solver64(cfg, _grid64(grid, origin, cell), float(np.float32(0.01)))
        got = []
        for k in range(case["scenes"]):
            part = slice(k * n, (k + 1) * n)
            goal, total = target[part].double(), case["scenes"] * n

            def loss(x, goal=goal, total=total):
                return ((x - goal) ** 2).sum() / total

            (p, v), gp, gv, gt = sol.gradients(pos[part].double(), vel[part].double(), loss)
            got.append((p, v, gp, gv, gt[None]))
        return dict(zip(("pos", "vel", "gpos", "gvel", "goffset"), (torch.cat(m) for m in zip(*got))))
    if kind == "mesh":
        _, f, moved = _deformed(case["subdiv"], seed)
        pts = np.random.default_rng(seed + 1).uniform([0.5, 0.0, 0.2], [1.1, 0.6, 0.8], (case["queries"], 3))
        rest = moved if case["rebuild"] else _deformed(case["subdiv"], seed)[0]
        dist = _mesh_grid64(moved, f, case["cell"], rest)[0]
        return {"dist": dist.reshape(-1), "face": None, "point": _mesh64(moved, f, pts.astype(np.float32))[1]}
    return None


def _mesh_grid64(verts, faces, cell, rest=None):
    """Signed distances at the voxels of the grid that the build over `rest` lays down: five cells around the
    mesh, voxel i at origin + i * cell."""
    box = np.asarray(verts if rest is None else rest)
    origin = box.min(0) - 5.0 * cell
    dims = np.ceil((box.max(0) + 5.0 * cell - origin) / cell).astype(int)
    axes = [torch.as_tensor(origin[a] + np.arange(dims[a]) * cell, device=DEV) for a in range(3)]
    pts = torch.stack(torch.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3)
    d, _, turn = _mesh64(verts, faces, pts.cpu().numpy())
    d = torch.where(turn.abs() > 0.5, -d, d)
    return d.reshape(*dims).cpu().numpy(), origin
