"""Batches of more scenes than get a warp each from the loop controllers (64), and of more than one
chunk of their block's threads (1,024): each scene against the same scene alone. The sums over a
scene's particles group their terms differently (1e-13), which can flip the last bit of a step
length, so states are held to 1e-6 of their norm after at most 5 iterations a solver, as in
test_gpu_halo.py."""
import numpy as np
import pytest

import vfd_gb300 as V
from vfd_gb300 import scenes

pytestmark = pytest.mark.gpu

ITER = ("PressureSolverIterationCount", "DivergenceSolverIterationCount", "ViscositySolverIterationCount")


def kinds():
    out = []
    for k, n in enumerate((1, 3, 4, 5, 6)):
        s = scenes.small_dam_break(n_side=n, r=0.01, viscosity=(0.0, 0.02)[k % 2])
        rng = np.random.default_rng(k)
        out.append(dict(s, v=rng.normal(0, 0.3, s["x"].shape).astype(np.float32),
                        desc=dict(s["desc"], MaxPressureSolverIterations=5, MaxDivergenceSolverIterations=5,
                                  MaxViscositySolverIterations=5)))
    return out


@pytest.mark.parametrize("count", [64, 65, 71, 1030])
def test_scenes_step_as_alone(count):
    sc = kinds()
    maps = [[V.build_box_map(b["min"], b["max"], b["inverted"], b["padding"], (8, 8, 8), 0.01) for b in s["boxes"]]
            for s in sc]
    alone = []
    for s, m in zip(sc, maps):
        sim = V.scene_simulation(s, maps=m)
        sim.Steps(2)
        alone.append((sim.GetDebugInfo(), sim.GetState()[:2]))
    batch = V.batch_simulation([sc[k % len(sc)] for k in range(count)], [maps[k % len(sc)] for k in range(count)])
    batch.Steps(2)
    for k in list(range(12)) + list(range(count - 12, count)):
        info, state = alone[k % len(sc)]
        got = batch.GetDebugInfo(k)
        for key in ITER:
            assert got[key] == info[key], (k, key)
        for a, b in zip(batch.GetState(k)[:2], state):
            assert np.linalg.norm(a - b) <= 1e-6 * max(np.linalg.norm(b), 1e-6), k
