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


def test_a_report_does_not_grow_with_the_scenes():
    """What a step brings back is the status and the first scene: a wait with nothing to do takes as long for
    4,096 scenes as for 16 (16 us; 210 where all scenes came back, so twice the smaller one leaves room)."""
    import time
    s = kinds()[1]

    def wait(count):
        sim = V.DFSPHSimulation(scenes=[V._abi.make_desc(**s["desc"])] * count)
        for k in range(count):
            sim.SetFluidObjects(s["x"], s["v"], scene=k)
        first = sim.OnUpdate()
        assert first["IterationCount"] == 1 and sim.GetDebugInfo(count - 1)["IterationCount"] == 1
        took = []
        for _ in range(30):
            t = time.perf_counter()
            sim.Synchronize()
            took.append(time.perf_counter() - t)
        return np.median(took)
    few, many = wait(16), wait(4096)
    assert many < 2.0 * few, (few, many)
