"""Four lanes a particle keep the sums of eight (two partial sums a lane, folded as the eight
are), so both give the same bits: rows of 0 to 70 neighbours, at the sizes around the line
where the default changes."""
import numpy as np
import pytest

import vfd_gb300 as V
from test_gpu_halo import block_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counts,tension,relative", [
    ((1, 1, 1), 0.0, False), ((3, 5, 11), 0.05, False), ((28, 29, 29), 0.05, False), ((29, 29, 29), 0.0, True)])
def test_four_lanes_are_eight(counts, tension, relative):
    s = block_scene(counts, tension)
    rng = np.random.default_rng(3)  # neighbours at all distances, and a knot at the neighbour cap
    x = s["x"] + rng.uniform(-0.004, 0.004, s["x"].shape).astype(np.float32)
    x[:200] = x[0] + rng.uniform(0.0, 0.01, x[:200].shape).astype(np.float32)
    s = dict(s, x=x, desc=dict(s["desc"], MaxPressureSolverIterations=4, MaxDivergenceSolverIterations=4,
                               MaxViscositySolverIterations=4))
    got = []
    for lanes in (4, 8):
        sim = V.scene_simulation(s)
        sim.SetPositionMode(relative)
        sim.SetLanes([lanes] * len(V.TUNED_KERNELS))
        sim.Steps(2)
        got.append([np.array(a) for a in sim.GetState()])
    for a, b in zip(*got):
        assert np.isfinite(a).all()
        np.testing.assert_array_equal(a, b)
