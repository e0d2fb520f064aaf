"""The narrow and the wide form of the staged tiles and the row kernels give the same bits: a run
that is waited for each step (the narrow form while few tiles outgrow it) against one launched at
once (after its first steps rows below 700,000 particles, the wide form above), from a lattice and
from states denser than the narrow form's halos, and against the row kernels with the bounds of
test_gpu_halo.py."""
import numpy as np
import pytest

from test_gpu_halo import assert_like_rows, block_scene
import vfd_gb300 as V

pytestmark = pytest.mark.gpu


def scene(counts, squeeze):
    s = block_scene(counts, 0.05)
    x = s["x"].copy()
    x *= np.float32(squeeze)
    return dict(s, x=x, desc=dict(s["desc"], MaxPressureSolverIterations=4, MaxDivergenceSolverIterations=4,
                                  MaxViscositySolverIterations=4))


@pytest.mark.parametrize("counts,squeeze,relative", [
    ((47, 48, 49), 1.0, False), ((47, 48, 49), 0.93, True), ((89, 90, 91), 1.0, True), ((89, 90, 91), 0.93, False),
    ((89, 90, 91), 0.88, False)])
def test_forms_agree(counts, squeeze, relative):
    s = scene(counts, squeeze)

    def make():
        sim = V.scene_simulation(s)
        sim.SetPositionMode(relative)
        return sim
    assert_like_rows(make)
    waited, queued = make(), make()
    for _ in range(10):
        waited.Steps(1)
    queued.Steps(10)
    for a, b in zip(waited.GetState(), queued.GetState()):
        assert np.isfinite(a).all()
        np.testing.assert_array_equal(a, b)
