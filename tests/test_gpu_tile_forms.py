"""The narrow and the wide form of the staged tiles give the same bits: a run that is waited for
each step (the narrow form while few tiles outgrow it) against one launched at once (the wide form
after the first steps), from a lattice and from a state denser than the narrow form's halos, and
against the row kernels with the bounds of test_gpu_halo.py."""
import numpy as np
import pytest

from test_gpu_halo import assert_like_rows, block_scene
import vfd_gb300 as V

pytestmark = pytest.mark.gpu


def scene(squeeze):
    s = block_scene((47, 48, 49), 0.05)
    x = s["x"].copy()
    x *= np.float32(squeeze)
    return dict(s, x=x, desc=dict(s["desc"], MaxPressureSolverIterations=4, MaxDivergenceSolverIterations=4,
                                  MaxViscositySolverIterations=4))


@pytest.mark.parametrize("squeeze", [1.0, 0.93, 0.88])
@pytest.mark.parametrize("relative", [False, True])
def test_forms_agree(squeeze, relative):
    s = scene(squeeze)

    def make():
        sim = V.scene_simulation(s)
        sim.SetPositionMode(relative)
        return sim
    assert_like_rows(make)
    waited, queued = make(), make()
    for _ in range(12):
        waited.Steps(1)
    queued.Steps(12)
    for a, b in zip(waited.GetState(), queued.GetState()):
        assert np.isfinite(a).all()
        np.testing.assert_array_equal(a, b)
