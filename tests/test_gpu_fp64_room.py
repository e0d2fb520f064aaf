"""The FP64 path where the GPU's memory does not hold the pairs' kept factors (1,120 bytes a particle):
it forms them again and steps as where they are kept, but for a rounding of a double here and there
(1e-13 of the values after two steps; the bound is test_gpu_fp64.py's 1e-9 h).
The memory is taken by plain allocations and given back."""
import numpy as np
import pytest

import vfd_gb300 as V
from vfd_gb300 import scenes

pytestmark = pytest.mark.gpu

MB = 1 << 20
N_SIDE = 60  # 216,000 particles: 242 MB of factors, 170 MB of other FP64 state


def drop():
    s = scenes.small_dam_break(n_side=N_SIDE, r=0.01, viscosity=0.02, surface_tension=0.05)
    x = s["x"]
    v = np.stack([np.sin(9 * x[:, 1]), np.cos(7 * x[:, 2]), np.sin(8 * x[:, 0])], 1).astype(np.float32)
    return dict(s, v=v, desc=dict(s["desc"], MaxDivergenceSolverIterations=4, MaxPressureSolverIterations=4,
                                  MaxViscositySolverIterations=6))


class Filled:
    """All of the GPU's free memory but about `left` bytes, held while inside."""

    def __init__(self, left):
        self.left = left

    def __enter__(self):
        import torch
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        self.held = []
        for piece in (1 << 32, 1 << 28, 1 << 24):
            while torch.cuda.mem_get_info()[0] - self.left >= piece:
                self.held.append(torch.empty(piece, dtype=torch.uint8, device="cuda"))
        return self

    def __exit__(self, *_):
        import torch
        self.held.clear()
        torch.cuda.empty_cache()


def simulation(s, analytic):
    sim = V.scene_simulation(s)
    sim.SetKernelMode(analytic)
    sim.Reset()  # the FP32 layout, before the memory goes
    return sim


@pytest.mark.parametrize("analytic", [False, True])
def test_without_room_for_the_pairs(analytic):
    s = drop()
    kept = simulation(s, analytic)
    kept.SetPrecision(True)
    kept.Steps(2)
    want = kept.GetStateF64()
    del kept
    sim = simulation(s, analytic)
    with Filled(256 * MB):
        sim.SetPrecision(True)
        sim.Steps(2)
        got = sim.GetStateF64()
    h = 4 * s["desc"]["ParticleRadius"]
    for a, b in zip(want, got):
        assert np.isfinite(b).all()
        assert np.abs(a - b).max() <= 1e-9 * h * max(1.0, np.abs(a).max())
    sim.Reset()  # with room again the factors are kept: the bits of the other run
    sim.Steps(2)
    for a, b in zip(want, sim.GetStateF64()):
        np.testing.assert_array_equal(a, b)


def test_a_refused_search_grid_leaves_no_cells_behind():
    # two particles 900 cells apart on each axis: 730 million cells, 8.7 GB
    s = scenes.small_dam_break(n_side=4, r=0.01)
    far = dict(s, x=s["x"].copy())
    far["x"][0] += np.float32(900 * 0.04)
    sim = V.scene_simulation(dict(s, boxes=[]))
    sim.SetPrecision(True)
    sim.Steps(1)
    want = sim.GetStateF64()
    sim.SetFluidObjects(far["x"], s["v"])
    sim.Reset()
    with Filled(1024 * MB):
        with pytest.raises(V.VFDError):
            sim.Steps(1)
    sim.SetFluidObjects(s["x"], s["v"])
    sim.Reset()  # the same particle count: the FP64 state serves again, with cells of its own
    sim.Steps(1)
    for a, b in zip(want, sim.GetStateF64()):
        np.testing.assert_array_equal(a, b)
