"""The staged-tile passes (layouts of 100,000 particles and more) against the FP32 oracle and
against the neighbour-row kernels, at the sizes and shapes where they can go wrong: ragged
blocks (part-filled tiles and warps), halos that outgrow the shared memory, tiles of a single
particle, rows longer than one round, and batches whose scenes end inside a tile's warp.

Tolerances. Against the oracle: those of one step from equal state in test_gpu_parity.py
(median 1e-6 h, maximum 1e-3 h; 0.05 h with surface tension, whose sampled coverage can flip).
Against the row kernels with eight lanes: the terms of each particle's sums, their order and
their rounding are the same, so densities and factors agree bit for bit; the sums over all
particles group their terms differently (1e-13), which can flip the last bit of a step length,
so velocities are held to 1e-6 of their norm after at most 5 iterations a solver.
"""
import numpy as np
import pytest

import vfd_gb300 as V
from vfd_gb300 import _abi, scenes
from test_gpu_parity import pair

pytestmark = pytest.mark.gpu

ITER = ("PressureSolverIterationCount", "DivergenceSolverIterationCount", "ViscositySolverIterationCount")
LANES8 = [8] * len(V.TUNED_KERNELS)


def block_scene(counts, tension, viscosity=0.05, r=0.005):
    s = scenes.viscous_dam_break(n_side=8, r=r)
    g = scenes.wall_gap(r)
    x = scenes.lattice_block(counts, r, (g, g, g), 0.05, scenes.SplitMix64(11))
    ext = [2.0 * r * c + 2.0 * g for c in counts]
    v = np.zeros_like(x)
    v[:, 0] = np.sin(20.0 * x[:, 1])
    v[:, 1] = np.cos(25.0 * x[:, 0])
    desc = dict(s["desc"], Viscosity=viscosity, EnableViscositySolver=int(viscosity > 0),
                SurfaceTension=tension, EnableSurfaceTensionSolver=int(tension > 0))
    return dict(s, x=x, v=v, desc=desc, boxes=[scenes.container((0, 0, 0), (2 * ext[0], 1.5 * ext[1], ext[2]), r, (20, 15, 10))])


@pytest.mark.parametrize("counts,tension,relative", [
    ((47, 48, 49), 0.0, False), ((50, 41, 53), 0.05, False), ((47, 48, 49), 0.0, True)])
def test_step_matches_oracle(counts, tension, relative):
    s = block_scene(counts, tension)
    assert len(s["x"]) >= 100000
    g, o = pair(s, 32)
    if relative:
        g.SetPositionMode(True)
    a, b = g.OnUpdate(), o.step()
    for k in ITER:
        assert abs(int(a[k]) - int(b[k])) <= 1, (k, a[k], b[k])
    h = 4 * s["desc"]["ParticleRadius"]
    dx = np.abs(g.GetState()[0] - o.state()[0]).max(axis=1)
    assert np.median(dx) < 1e-6 * h * (10 if relative else 1) and dx.max() < (0.05 if tension else 1e-3) * h, \
        (np.median(dx) / h, dx.max() / h)


def assert_like_rows(make):
    tiles, rows = make(), make()
    rows.SetLanes(LANES8)
    a, b = tiles.OnUpdate(), rows.OnUpdate()
    for k in ITER + ("MaxNeighborCount",):
        assert a[k] == b[k], (k, a[k], b[k])
    if tiles.scene_count == 1:
        np.testing.assert_array_equal(tiles.GetField(_abi.FIELD_DENSITY), rows.GetField(_abi.FIELD_DENSITY))
    for scene in range(tiles.scene_count):
        for u, w in zip(tiles.GetState(scene)[:2], rows.GetState(scene)[:2]):
            assert np.isfinite(u).all()
            assert np.linalg.norm(u - w) <= 1e-6 * max(np.linalg.norm(w), 1e-6), scene


@pytest.mark.parametrize("relative", [False, True])
def test_crowded_halos_and_lone_particles(relative):
    # a block at rest spacing, a cluster of three times its density (halos of ~3,500 particles,
    # the neighbour cap) and particles two cells and more apart from everything
    s = block_scene((46, 47, 48), 0.05)
    r = s["desc"]["ParticleRadius"]
    h = 4 * r
    rng = np.random.default_rng(5)
    cluster = (np.array([0.75, 0.2, 0.2]) + 5 * h * rng.random((3000, 3))).astype(np.float32)
    lone = (np.array([0.6, 0.55, 0.1]) + 3 * h * np.stack(np.meshgrid(*[np.arange(4)] * 3), -1).reshape(-1, 3)).astype(np.float32)
    x = np.concatenate([s["x"], cluster, lone])
    v = np.concatenate([s["v"], np.zeros_like(cluster), np.zeros_like(lone)]).astype(np.float32)
    s = dict(s, x=x, v=v, desc=dict(s["desc"], MaxPressureSolverIterations=5, MaxDivergenceSolverIterations=5,
                                    MaxViscositySolverIterations=5))

    def make():
        sim = V.scene_simulation(s)
        if relative:
            sim.SetPositionMode(True)
        return sim
    assert_like_rows(make)


def test_batch_of_uneven_scenes():
    sizes = [(47, 46, 45), (1, 1, 1), (3, 5, 2), (20, 20, 21), (9, 31, 7)]
    sc = [block_scene(c, 0.05 if k % 2 else 0.0, viscosity=0.0 if k == 3 else 0.05) for k, c in enumerate(sizes)]
    for s in sc:
        s["desc"].update(MaxPressureSolverIterations=5, MaxDivergenceSolverIterations=5, MaxViscositySolverIterations=5)
    assert sum(len(s["x"]) for s in sc) >= 100000
    maps = [[V.build_box_map(b["min"], b["max"], b["inverted"], b["padding"], b["resolution"], 0.005) for b in s["boxes"]]
            for s in sc]
    assert_like_rows(lambda: V.batch_simulation(sc, maps))
