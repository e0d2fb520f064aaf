"""Performance cases of the DFSPH framework: what is timed, on which inputs.

Each case is one call sequence a program makes through the public Python entry points.
The step is measured the way a coupled program drives it: the handle (buffers, volume maps,
step graphs) is kept, each pass brings positions and velocities from pinned host memory,
advances, and reads positions, velocities and accelerations back. A pass takes the other
one of two velocity fields than the pass before: with the same one the viscosity solve
would start from its own solution.

  kind "step"     SetState, Steps, GetStateInto of a scene: "block" (a dam break in a
                  closed box), "drop" (a viscous drop in free fall) or "jet" (a viscous jet
                  above a resting pool)
  kind "batch"    Reset, Steps, GetStateInto of independent scenes advanced together
  kind "adjoint"  SetState, AdjointForward, GetStateInto, AdjointBackward of a drop
  kind "fp64"     Reset, Steps, GetStateF64 of a drop on the FP64 path
  kind "search"   the allocation-free neighbour search on device buffers
  kind "legacy"   Reset, SetVelocities, Steps, GetState of the legacy SPH solver
  kind "map"      the volume map of a triangle mesh
"""
import math

import numpy as np
import torch

import vfd_gb300 as V
from vfd_gb300 import _abi, meshes, sph
from vfd_gb300.scenes import SOLVER

VISCOUS = dict(EnableViscositySolver=1, MaxViscositySolverError=0.01)


def listed():
    return [
        # the smallest call: neighbours of a few thousand device-resident points, launches only
        dict(name="search_4k", kind="search", n=4096),
        # the 8,000-particle dam break (inviscid, no surface tension), an interactive scene
        dict(name="dam_break_8k", kind="step", scene="block", nx=20, ny=20, nz=20, r=0.025, viscosity=0.0,
             tension=0.0, relative=False, steps=1),
        # the 33k viscous drop, forward
        dict(name="drop_33k", kind="step", scene="drop", n=33401, r=0.0025, viscosity=0.01, tension=0.0,
             relative=False, steps=1),
        # the same drop differentiated, on the smooth kernel with a fixed time step as gradients are taken in
        # earnest: recorded forward run with one replayed segment, and backward
        dict(name="adjoint_33k", kind="adjoint", n=33401, r=0.0025, viscosity=0.01, steps=4, every=2),
        # the FP64 path, the trajectory that the FP32 ones are checked against
        dict(name="fp64_drop_8k", kind="fp64", n=8217, r=0.004, viscosity=0.01, steps=2),
        # cell-relative positions (scenes far from the origin), viscosity and surface tension
        dict(name="dam_relative_64k", kind="step", scene="block", nx=41, ny=39, nz=40, r=0.005, viscosity=0.05,
             tension=0.05, relative=True, steps=1),
        # scenes of uneven size and viscosity advanced together, as a parameter sweep does
        dict(name="batch_48", kind="batch", scenes=48, n_min=2000, n_max=64000, steps=1),
        # the 1M-particle high-viscosity dam break with surface tension, the headline workload
        dict(name="viscous_dam_1m", kind="step", scene="block", nx=100, ny=100, nz=100, r=0.005, viscosity=0.05,
             tension=0.05, relative=False, steps=1),
        # the 8M-particle jet above its pool, the largest configuration
        dict(name="jet_8m", kind="step", scene="jet", nx=400, ny=50, nz=400, r=0.0015, viscosity=0.2,
             tension=1.51e-5, relative=False, steps=1),
        # the legacy solver at the size of an interactive scene
        dict(name="legacy_262k", kind="legacy", nx=64, ny=64, nz=64, steps=20),
        # scene set-up: the volume map of a mesh, at the default resolution
        dict(name="mesh_map_20", kind="map", subdivisions=4, rx=20, ry=20, rz=20),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "search", "batch", "adjoint", "fp64", "legacy", "map"])
    if kind == "step":
        scene = rng.choice(["block", "block", "drop", "jet"])
        if scene == "drop":
            return dict(kind=kind, scene=scene, n=_log_int(rng, 2000, 300000), r=0.0025,
                        viscosity=math.exp(rng.uniform(math.log(0.001), math.log(0.1))), tension=0.0,
                        relative=rng.random() < 0.3, steps=1)
        if scene == "jet":
            side = _log_int(rng, 100, 330)
            return dict(kind=kind, scene=scene, nx=side, ny=rng.randint(20, 50), nz=side + rng.randint(-9, 9), r=0.0015,
                        viscosity=0.2, tension=1.51e-5, relative=rng.random() < 0.5, steps=1)
        side = _log_int(rng, 12, 120)
        viscous = rng.random() < 0.7
        return dict(kind=kind, scene=scene, nx=side, ny=max(8, side + rng.randint(-7, 7)),
                    nz=max(8, side + rng.randint(-7, 7)), r=0.005,
                    viscosity=math.exp(rng.uniform(math.log(0.005), math.log(0.1))) if viscous else 0.0,
                    tension=0.05 if viscous and rng.random() < 0.5 else 0.0, relative=rng.random() < 0.3, steps=1)
    if kind == "search":
        return dict(kind=kind, n=_log_int(rng, 500, 16384))
    if kind == "batch":
        return dict(kind=kind, scenes=rng.randint(8, 64), n_min=2000, n_max=_log_int(rng, 8000, 64000), steps=1)
    if kind == "adjoint":
        return dict(kind=kind, n=_log_int(rng, 2000, 60000), r=0.0025, viscosity=0.01, steps=rng.randint(1, 5),
                    every=rng.randint(1, 3))
    if kind == "fp64":
        return dict(kind=kind, n=_log_int(rng, 1000, 30000), r=0.004, viscosity=0.01, steps=1)
    if kind == "legacy":
        side = _log_int(rng, 16, 90)
        return dict(kind=kind, nx=side, ny=side + rng.randint(-3, 3), nz=side + rng.randint(-3, 3), steps=20)
    return dict(kind="map", subdivisions=rng.randint(2, 5), rx=rng.randint(8, 32), ry=rng.randint(8, 32),
                rz=rng.randint(8, 32))


# ---------------------------------------------------------------- inputs, from the seed alone
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _lattice(nx, ny, nz, spacing, origin):
    ax = [torch.arange(k, device="cuda", dtype=torch.float64) * spacing + o for k, o in zip((nx, ny, nz), origin)]
    return torch.stack(torch.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)


def _jitter(x, amount, g):
    return x + (2.0 * torch.rand(x.shape, generator=g, device="cuda", dtype=torch.float64) - 1.0) * amount


def _flow(x, extent, speed, g):
    """A smooth velocity field of eight Fourier modes with the largest speed `speed`."""
    p = torch.rand(8, 7, generator=g, device="cuda", dtype=torch.float64)
    v = torch.zeros_like(x)
    for m in range(8):
        k = (2.0 * math.pi / extent) * (1.0 + 2.0 * p[m, 0])
        z = 2.0 * p[m, 1] - 1.0
        s = torch.sqrt(1.0 - z * z)
        d = torch.stack([s * torch.cos(2 * math.pi * p[m, 2]), s * torch.sin(2 * math.pi * p[m, 2]), z])
        v += torch.sin(x @ (k * d) + 2.0 * math.pi * p[m, 6])[:, None] * (2.0 * p[m, 3:6] - 1.0)
    return v * (speed / v.norm(dim=1).max().clamp_min(1e-12))


def _pinned(t):
    h = torch.empty(t.shape, dtype=torch.float32, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _sphere(n, r, center):
    """About n lattice points (spacing 2r) of a sphere."""
    radius = 2.0 * r * (3.0 * n / (4.0 * math.pi)) ** (1.0 / 3.0)
    m = int(radius / (2.0 * r)) + 1
    x = _lattice(2 * m + 1, 2 * m + 1, 2 * m + 1, 2.0 * r, (-2.0 * r * m,) * 3)
    x = x[(x * x).sum(1) <= radius * radius]
    return x + torch.tensor(center, device="cuda", dtype=torch.float64), radius


def _drop(n, r, g):
    radius = 2.0 * r * (3.0 * n / (4.0 * math.pi)) ** (1.0 / 3.0)
    c = (3.0 * radius, 3.5 * radius, 3.0 * radius)
    x, _ = _sphere(n, r, c)
    x = _jitter(x, 0.1 * r, g)
    box = dict(min=(0.0, 0.0, 0.0), max=(6.0 * radius, 0.5 * radius, 6.0 * radius), inverted=False, resolution=(20, 8, 20))
    return x, _flow(x, 2.0 * radius, 0.5, g), box


def _block(nx, ny, nz, r, g):
    x = _jitter(_lattice(nx, ny, nz, 2.0 * r, (3.0 * r,) * 3), 0.1 * r, g)
    ext = [2.0 * r * k + 4.0 * r for k in (nx, ny, nz)]
    box = dict(min=(0.0, 0.0, 0.0), max=(2.0 * ext[0], 1.5 * ext[1], ext[2]), inverted=True, resolution=(40, 30, 20))
    return x, _flow(x, 0.5 * max(ext), 0.75, g), box


def _jet(nx, ny, nz, r, g):
    x, v, box = _block(nx, ny, nz, r, g)
    box = dict(box, max=(2.0 * r * nx + 4.0 * r, 2.0 * r * ny + 0.6, 2.0 * r * nz + 4.0 * r), resolution=(40, 24, 40))
    top, m = 2.0 * r * ny + 8.0 * r, int(0.02 / (2.0 * r))
    col = _lattice(2 * m + 1, int(0.3 / (2.0 * r)), 2 * m + 1, 2.0 * r, (-2.0 * r * m, top, -2.0 * r * m))
    col = col[col[:, 0] ** 2 + col[:, 2] ** 2 <= 0.02 ** 2]
    col = _jitter(col, 0.02 * r, g) + torch.tensor((0.5 * box["max"][0], 0.0, 0.5 * box["max"][2]), device="cuda",
                                                   dtype=torch.float64)
    vc = torch.zeros_like(col)
    vc[:, 1] = -1.0
    return torch.cat([x, col]), torch.cat([0.1 * v, vc]), box


def _desc(c):
    more = dict(MaxTimeStepSize=0.001) if c["kind"] == "adjoint" else {}
    return _abi.make_desc(ParticleRadius=c["r"], Viscosity=c["viscosity"], BoundaryViscosity=c["viscosity"],
                          SurfaceTension=c.get("tension", 0.0), EnableSurfaceTensionSolver=int(c.get("tension", 0.0) > 0),
                          **{**VISCOUS, "EnableViscositySolver": int(c["viscosity"] > 0), **SOLVER, **more})


def _map(box, r):
    return V.build_box_map(box["min"], box["max"], box["inverted"], 0.0, box["resolution"], r)


def _scene(c, seed):
    g = _generator(seed)
    if c.get("scene", "drop") == "drop":
        return _drop(c["n"], c["r"], g)
    return (_jet if c["scene"] == "jet" else _block)(c["nx"], c["ny"], c["nz"], c["r"], g)


def _simulation(c, x, v, box):
    sim = V.DFSPHSimulation(_desc(c))
    sim.SetFluidObjects(x, v)
    sim.AddRigidBody(_map(box, c["r"]))
    if c["kind"] == "adjoint":
        sim.SetKernelMode(True)
    if c.get("relative"):
        sim.SetPositionMode(True)
    return sim


def _batch(c, seed):
    """(description, positions, velocities, box) of each scene: blocks and drops in turn."""
    g = _generator(seed)
    out = []
    for k in range(c["scenes"]):
        # sizes and viscosities log-uniform, a low-discrepancy sequence (the same for every seed)
        u = (0.5 + k * 0.7548776662466927) % 1.0, (0.5 + k * 0.5698402909980532) % 1.0
        n = c["n_min"] * (c["n_max"] / c["n_min"]) ** u[0]
        d = dict(kind="batch", r=0.005, viscosity=1e-5 * 1e4 ** u[1])
        side = max(4, int(round(n ** (1.0 / 3.0))))
        x, v, box = _block(side, max(4, int(n / side ** 2)), side, 0.005, g) if k % 2 == 0 else _drop(n, 0.005, g)
        out.append((_desc(d), x.float().cpu().numpy(), v.float().cpu().numpy(), dict(box, resolution=(16, 16, 16))))
    return out


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("step", "adjoint", "fp64"):
        x, v, box = _scene(c, seed)
        other = v.flip(1)  # the same field along other axes, as smooth and as fast
        x, v = _pinned(x), _pinned(v)
        state = dict(case=c, x=x, v=[v, _pinned(other)], turn=0, sim=_simulation(c, x, v, box))
        if kind == "fp64":
            state["sim"].SetPrecision(True)
            return state
        state["sim"].Reset()
        state["out"] = tuple(_pinned(torch.zeros(x.shape)) for _ in range(3))
        if kind == "adjoint":
            g = _generator(seed + 7919)
            state["bar"] = [_pinned(torch.randn(x.shape, generator=g, device="cuda") / len(x)) for _ in range(2)]
        return state
    if kind == "batch":
        scenes = _batch(c, seed)
        sim = V.DFSPHSimulation(scenes=[s[0] for s in scenes])
        for k, (_, x, v, box) in enumerate(scenes):
            sim.SetFluidObjects(x, v, scene=k)
            sim.AddRigidBody(_map(box, 0.005), scene=k)
        ends = np.cumsum([0] + [len(s[1]) for s in scenes])
        out = tuple(_pinned(torch.zeros(int(ends[-1]), 3)) for _ in range(3))
        return dict(case=c, sim=sim, out=out, ends=[int(e) for e in ends])
    if kind == "search":
        side = int(round(c["n"] ** (1.0 / 3.0))) + 1
        x = _jitter(_lattice(side, side, side, 0.05, (0.0, 0.0, 0.0)), 0.01, _generator(seed))[:c["n"]]
        new = lambda *s: torch.zeros(*s, dtype=torch.int32, device="cuda")  # noqa: E731
        return dict(case=c, x=x.float().contiguous(), counts=new(c["n"]), rows=new(c["n"], _abi.MAX_NEIGHBORS),
                    order=new(c["n"]))
    if kind == "legacy":
        g = _generator(seed)
        half = [0.5 * 0.004 * k for k in (c["nx"], c["ny"], c["nz"])]
        x = _jitter(_lattice(c["nx"], c["ny"], c["nz"], 0.004, [-h for h in half]), 0.0004, g)
        v = _flow(x, 2.0 * max(half), 0.3, g)
        lim = [h + 0.1 for h in half]
        d = sph.make_sph_desc(WorldMin=[-h for h in lim], WorldMax=lim)
        return dict(case=c, v=_pinned(v), sim=sph.SPHSimulation(d, x.float().cpu().numpy()))
    verts, tris = meshes.icosphere((0.0, 0.0, 0.0), 0.5, c["subdivisions"])
    p = torch.rand(3, generator=_generator(seed), device="cuda", dtype=torch.float64).cpu().numpy()
    verts = (verts.astype(np.float64) * (0.6 + 0.4 * p) + 0.1 * p).astype(np.float32)  # an ellipsoid
    return dict(case=c, verts=verts, tris=tris)


# ---------------------------------------------------------------- one pass
def run(state):
    c, kind = state["case"], state["case"]["kind"]
    sim = state.get("sim")
    if kind in ("step", "adjoint"):
        sim.SetState(state["x"], state["v"][state["turn"] % 2])
        state["turn"] += 1
    if kind == "step":
        sim.Steps(c["steps"])
        sim.GetStateInto(*state["out"])
        return state["out"]
    if kind == "adjoint":
        sim.AdjointForward(c["steps"], c["every"])
        sim.GetStateInto(*state["out"])
        return state["out"] + sim.AdjointBackward(*state["bar"])
    if kind == "fp64":
        sim.Reset()
        sim.Steps(c["steps"])
        return sim.GetStateF64()
    if kind == "batch":
        sim.Reset()
        sim.Steps(c["steps"])
        for k, (a, b) in enumerate(zip(state["ends"], state["ends"][1:])):
            sim.GetStateInto(*(o[a:b] for o in state["out"]), scene=k)
        return state["out"]
    if kind == "search":
        V.find_neighbors_noalloc(state["x"].data_ptr(), c["n"], 0.025, state["counts"].data_ptr(),
                                 state["rows"].data_ptr(), state["order"].data_ptr())
        return state["counts"], state["rows"], state["order"]
    if kind == "legacy":
        sim.Reset()
        sim.SetVelocities(state["v"])
        sim.Steps(c["steps"])
        return sim.GetState()
    m = V.build_mesh_map(state["verts"], state["tris"], None, False, 0.0, (c["rx"], c["ry"], c["rz"]), 0.025)
    n = m.struct.node_count
    return m.nodes[:n], m.nodes[n:], m.cells, m.cell_map


# ---------------------------------------------------------------- work
def work(case):
    c, kind = case, case["kind"]
    if kind == "map":
        nodes = (c["rx"] + 1) * (c["ry"] + 1) * (c["rz"] + 1) + 2 * (
            c["rx"] * (c["ry"] + 1) * (c["rz"] + 1) + (c["rx"] + 1) * c["ry"] * (c["rz"] + 1)
            + (c["rx"] + 1) * (c["ry"] + 1) * c["rz"])
        cells = c["rx"] * c["ry"] * c["rz"]
        faces = 20 * 4 ** c["subdivisions"]
        # the nearest face of a node through a hierarchy over the faces, and 16^3 quadrature points of ~100
        # operations at the nodes within the support of the surface (a fifth of them)
        return dict(bytes=8 * nodes + 8 * 33 * cells + 24 * faces, flops=nodes * (60 * math.log2(faces) + 0.2 * 4096 * 100))
    if kind == "search":
        return dict(bytes=c["n"] * (12 + 8 + 4 * 30), flops=c["n"] * 216 * 8)
    n = {"jet": lambda: c["nx"] * c["ny"] * c["nz"] + 15618, "block": lambda: c["nx"] * c["ny"] * c["nz"],
         "drop": lambda: c["n"]}[c.get("scene", "block" if kind == "legacy" else "drop")]() if kind != "batch" else \
        int(c["scenes"] * (c["n_max"] - c["n_min"]) / math.log(c["n_max"] / c["n_min"]))
    if kind == "legacy":
        return dict(bytes=n * (12 + c["steps"] * 64 + 32), flops=n * c["steps"] * 30 * 40)
    # a step: the carried state (x, v, warm start, curvature) read and written once; thirty pairs a particle in
    # every neighbour pass (search, density, two iterations of two passes for either pressure solve with their
    # first and last passes, and for viscosity its set-up and ten products)
    viscous = c.get("viscosity", 1.0) > 0
    passes = 2 + 2 * (2 * 2 + 2) + (12 if viscous else 0) + (2 if c.get("tension", 0.0) > 0 else 0)
    word = 8 if kind == "fp64" else 4
    steps = c["steps"] * (3 if kind == "adjoint" else 1)
    return dict(bytes=n * (60 + steps * 20 * word), flops=n * steps * passes * 30 * 20)


# ---------------------------------------------------------------- 64-bit values
def exact(case, seed):
    """The drop's step (no wall in reach) and the mesh distances in 64 bits. A step near walls, with surface
    tension's sampled normals, its derivative, and the legacy solver's stiff walls have no plain statement
    of this length; a search returns whole numbers."""
    if case["kind"] == "map":
        return _exact_map(case, seed)
    if case["kind"] not in ("step", "fp64") or case.get("scene", "drop") != "drop" or case.get("n") > 40000:
        return None
    x, v, _ = _scene(case, seed)
    x, v, a = _exact_drop(case, x.float().double(), v.float().double())
    return (x, v) if case["kind"] == "fp64" else (x, v, a)


def _exact_drop(case, x, v):
    """Steps of the method in 64 bits for particles far from every wall: cubic spline tables of 10,000 entries
    read at the middle of an entry, two Jacobi pressure solves, the block-Jacobi CG of the viscosity."""
    d = _desc(case)
    n, r0 = len(x), d.ParticleRadius
    h, rho0, vol = 4.0 * r0, 1000.0, 0.8 * (2.0 * r0) ** 3
    mass, cmu, eps2 = vol * rho0, 10.0 * d.Viscosity * rho0, 0.01 * h * h
    step = h / 9999.0
    q = torch.arange(10000, device="cuda", dtype=torch.float64) / 9999.0
    kw, kg = 8.0 / (math.pi * h ** 3), 48.0 / (math.pi * h ** 3)
    tw = torch.where(q <= 0.5, kw * (6.0 * q ** 3 - 6.0 * q ** 2 + 1.0), kw * 2.0 * (1.0 - q) ** 3)
    tg = torch.where(q <= 0.5, kg * (3.0 * q - 2.0) / (h * h), -kg * (1.0 - q) ** 2 / (q.clamp_min(1e-9) * h * h))
    tg[0] = 0.0
    tw, tg = 0.5 * (tw[:-1] + tw[1:]), 0.5 * (tg[:-1] + tg[1:])
    dt, dv = float(d.TimeStepSize), torch.zeros_like(x)
    gravity = torch.tensor(list(d.Gravity), device="cuda", dtype=torch.float64)
    for _ in range(case["steps"]):
        i, j = [], []
        for b in range(0, n, 2048):
            near = ((x[b:b + 2048, None, :] - x[None, :, :]) ** 2).sum(-1)
            p = torch.nonzero((near < h * h) & (near > 0.0))
            i.append(p[:, 0] + b)
            j.append(p[:, 1])
        i, j = torch.cat(i), torch.cat(j)
        r = x[i] - x[j]
        r2 = (r * r).sum(1)
        at = (r2.sqrt() / step).long().clamp_max(9998)
        gs = tg[at]
        g = gs[:, None] * r

        def total(t):
            return torch.zeros((n,) + t.shape[1:], device="cuda", dtype=torch.float64).index_add_(0, i, t)

        count = total(torch.ones_like(r2))
        rho = rho0 * vol * (kw + total(tw[at]))
        den = vol * vol * (total((g * g).sum(1)) + (total(g) ** 2).sum(1))
        alpha = torch.where(den > 1e-5, 1.0 / den, torch.zeros_like(den))

        def divergence(w):
            return vol * total(((w[i] - w[j]) * g).sum(1))

        def force(k):
            s = k[i] + k[j]
            s = torch.where(s.abs() > 1e-5, s, torch.zeros_like(s))
            return total((-vol * s)[:, None] * g)

        def solve(k, al, source, scale, least, most, eta, few):
            it, err = 0, 0.0
            while (err > eta or it < least) and it < most:
                res = (source - divergence(force(k)) * scale).clamp_max(0.0)
                res = torch.where(few, torch.zeros_like(res), res)
                k = k - res * al
                err = -rho0 * float(res.sum()) / n
                it += 1
            return k

        few = count < 20
        adv = torch.where(few, torch.zeros_like(rho), divergence(v).clamp_min(0.0))
        k = solve(adv * alpha / dt, alpha / dt, -adv, dt, d.MinDivergenceSolverIterations,
                  d.MaxDivergenceSolverIterations, d.MaxDivergenceSolverError * 1e-4 * rho0 / dt, few)
        v = v + dt * force(k)
        acc = gravity.expand_as(x)

        c = cmu * mass / rho[j] / (r2 + eps2)
        eye = torch.eye(3, device="cuda", dtype=torch.float64)
        inv = torch.linalg.inv(eye - (dt / rho)[:, None, None] * total(c[:, None, None] * r[:, :, None] * g[:, None, :]))

        def apply(w):
            return w - (dt / rho)[:, None] * total((c * ((w[i] - w[j]) * r).sum(1))[:, None] * g)

        w = v + dv
        res = v - apply(w)
        stop = max(d.MaxViscositySolverError ** 2 * 1e-4 * float((v * v).sum()), 1.1754944e-38)
        if float((res * res).sum()) >= stop:
            p = torch.einsum("nij,nj->ni", inv, res)
            rz = abs(float((res * p).sum()))
            for _ in range(d.MaxViscositySolverIterations):
                ap = apply(p)
                al = rz / float((p * ap).sum())
                w, res = w + al * p, res - al * ap
                if float((res * res).sum()) < stop:
                    break
                z = torch.einsum("nij,nj->ni", inv, res)
                old, rz = rz, abs(float((res * z).sum()))
                p = z + (rz / old) * p
        dv = w - v
        acc = acc + dv / dt
        top = max(0.1, float(((v + acc * dt) ** 2).sum(1).max()))
        dt = max(min(0.4 * 2.0 * r0 / math.sqrt(top), d.MaxTimeStepSize), d.MinTimeStepSize)
        v = v + dt * acc
        adv = rho / rho0 + dt * divergence(v)
        k = solve((adv - 1.0).clamp_min(0.0) * alpha / dt ** 2, alpha / dt ** 2, 1.0 - adv, dt * dt,
                  d.MinPressureSolverIterations, d.MaxPressureSolverIterations, d.MaxPressureSolverError * 1e-4 * rho0,
                  torch.zeros_like(few))
        v = v + dt * force(k)
        x = x + dt * v
    return x, v, acc


def _exact_map(case, seed):
    """Signed distance to the mesh at the nodes of the map's grid (corners, then two points on each edge)."""
    s = prepare(case, seed)
    res = (case["rx"], case["ry"], case["rz"])
    verts = torch.from_numpy(s["verts"]).cuda().double()
    a, b, c = (verts[torch.from_numpy(s["tris"][:, k].astype(np.int64)).cuda()] for k in range(3))
    margin = 32.0 * 0.025 - 0.025  # the map reaches eight support radii, less the tolerance, past the mesh
    lo = verts.amin(0) - margin
    cs = (verts.amax(0) + margin - lo) / torch.tensor(res, device="cuda", dtype=torch.float64)

    def axis(k, edge):
        return torch.arange(res[k] + (0 if edge else 1), device="cuda", dtype=torch.float64)

    pts = []
    z, y, x = torch.meshgrid(axis(2, 0), axis(1, 0), axis(0, 0), indexing="ij")
    pts.append(torch.stack([x, y, z], -1).reshape(-1, 3))
    for e, order in ((0, (2, 1, 0)), (1, (0, 2, 1)), (2, (1, 0, 2))):
        grids = torch.meshgrid(*(axis(k, k == e) for k in order), indexing="ij")
        base = torch.stack([grids[order.index(k)] for k in range(3)], -1).reshape(-1, 1, 3).repeat(1, 2, 1)
        base[:, 0, e] += 1.0 / 3.0
        base[:, 1, e] += 2.0 / 3.0
        pts.append(base.reshape(-1, 3))
    p = torch.cat(pts) * cs + lo
    if len(p) * len(a) > 4e8:
        return None
    n = torch.linalg.cross(b - a, c - a)
    n = n / n.norm(dim=1, keepdim=True)
    out = []
    for k in range(0, len(p), 4096):
        q = p[k:k + 4096, None, :]
        best = torch.full((q.shape[0], len(a)), math.inf, device="cuda", dtype=torch.float64)
        inside = torch.ones_like(best, dtype=torch.bool)
        for u, w in ((a, b), (b, c), (c, a)):
            e = w - u
            t = (((q - u) * e).sum(-1) / (e * e).sum(-1)).clamp(0.0, 1.0)
            best = torch.minimum(best, ((q - u - t[..., None] * e) ** 2).sum(-1))
            inside &= (torch.linalg.cross(e, n)[None] * (q - u)).sum(-1) <= 0.0
        plane = ((q - a) * n).sum(-1)
        best = torch.where(inside, plane * plane, best)
        dist = best.amin(1).sqrt()
        # a convex mesh: a point is inside when it lies behind every face's plane
        out.append(torch.where((plane <= 0.0).all(1), -dist, dist))
    # field 0 is the distance less the collision tolerance (padding - radius = -radius)
    return torch.cat(out) + 0.025, None, None, None
