"""Layouts where the GPU's memory is short: the buffers that a layout can do without (the tiles' lists, the
kept start) give way to those that it needs, and a read of the state, which borrows scratch of the
step, changes nothing."""
import numpy as np
import pytest

from test_gpu_fp64_room import Filled
from test_gpu_halo import block_scene
import vfd_gb300 as V

pytestmark = pytest.mark.gpu


def scene():
    s = block_scene((117, 117, 117), 0.05)  # 1.6M particles
    return dict(s, desc=dict(s["desc"], MaxPressureSolverIterations=4, MaxDivergenceSolverIterations=4,
                             MaxViscositySolverIterations=4))


def used_by(make):
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    sim = make()
    return sim, before - torch.cuda.mem_get_info()[0]


def test_a_layout_without_its_spare_buffers():
    s = scene()

    def make():
        sim = V.scene_simulation(s)
        sim.Reset()
        return sim
    sim, full = used_by(make)
    spare = (32 + 24) * len(s["x"])  # the lists of the halos, 51 MB, and the kept start, 38
    sim.SetTileForm(0)
    sim.Steps(2)
    want = sim.GetState()
    del sim
    with Filled(full - spare):  # and up to 16 MB more: room for neither
        sim = make()
        for _ in range(2):
            sim.Steps(2)
            assert sim.TileForm() == 0
            for a, b in zip(want, sim.GetState()):
                np.testing.assert_array_equal(a, b)
            sim.Reset()


def test_reading_between_steps_changes_nothing():
    sims = [V.scene_simulation(scene()) for _ in range(2)]
    for _ in range(3):
        sims[0].Steps(1)
        sims[0].GetState()
        sims[1].Steps(1)
    for a, b in zip(*(sim.GetState() for sim in sims)):
        np.testing.assert_array_equal(a, b)
