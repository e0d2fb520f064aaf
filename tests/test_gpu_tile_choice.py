"""Each step takes the form of the staged tiles that its own state asks for: narrow on a lattice,
rows (below 700,000 particles) or wide tiles on denser fluid, however the state came about (set,
restored, queued, launched by the host) and whatever ran before it."""
import numpy as np
import pytest

from test_gpu_halo import block_scene
import vfd_gb300 as V

pytestmark = pytest.mark.gpu

SMALL, LARGE = (47, 48, 49), (89, 90, 91)
ROWS, NARROW, WIDE = 0, 1, 2


def scene(counts, squeeze=1.0):
    # squeezed to 0.88 of the spacing, a cell holds 11.7 particles: tiles of 376, beyond the narrow form
    s = block_scene(counts, 0.05)
    return dict(s, x=s["x"] * np.float32(squeeze), v=0 * s["v"],
                desc=dict(s["desc"], MaxPressureSolverIterations=3, MaxDivergenceSolverIterations=3,
                          MaxViscositySolverIterations=3))


@pytest.mark.parametrize("counts,other", [(SMALL, ROWS), (LARGE, WIDE)])
def test_set_states(counts, other):
    s, dense = scene(counts), scene(counts, 0.88)
    sim = V.scene_simulation(s)
    for state, form in ((s, NARROW), (dense, other), (dense, other), (s, NARROW)):
        sim.SetState(state["x"], state["v"])
        sim.Steps(1)
        assert sim.TileForm() == form
    sim.SetState(dense["x"], dense["v"])
    sim.StepsAsync(2)
    sim.Synchronize()
    assert sim.TileForm() == other
    sim.Reset()
    sim.Steps(12)
    assert sim.TileForm() == NARROW  # the lattice at rest, in every queued step


def test_start_and_restore_of_dense_fluid():
    dense = V.scene_simulation(scene(SMALL, 0.88))
    dense.Steps(1)
    assert dense.TileForm() == ROWS
    image = dense.Checkpoint()
    sim = V.scene_simulation(scene(SMALL))
    sim.Restore(image)
    dense.Steps(2)
    sim.Steps(2)
    assert sim.TileForm() == dense.TileForm() == ROWS
    for a, b in zip(dense.GetState(), sim.GetState()):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("squeeze,form", [(1.0, NARROW), (0.88, ROWS)])
def test_launched_by_the_host(squeeze, form):
    graph, host = (V.scene_simulation(scene(SMALL, squeeze)) for _ in range(2))
    host.SetGraphMode(False)
    for sim in (graph, host):
        sim.Steps(2)
        assert sim.TileForm() == form
    assert graph.GetGraphMode() == (True, True)
    for a, b in zip(graph.GetState(), host.GetState()):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("counts,other", [((64, 64, 64), ROWS), (LARGE, WIDE)])
@pytest.mark.parametrize("tuned_on_lattice", [True, False])
def test_tuning_keeps_the_forms_it_does_not_find_slower(counts, other, tuned_on_lattice):
    # the narrow form takes 2,705 us a step of 260,000 particles on a lattice, rows 3,027; at
    # 729,000 the lines lie further apart
    s, dense = scene(counts), scene(counts, 0.88)
    sim = V.scene_simulation(s if tuned_on_lattice else dense)
    before = sim.GetState()
    sim.Autotune(2)
    for a, b in zip(before, sim.GetState()):
        np.testing.assert_array_equal(a, b)
    sim.SetState(s["x"], s["v"])
    sim.Steps(1)
    assert sim.TileForm() == NARROW
    sim.SetState(dense["x"], dense["v"])
    sim.Steps(1)
    assert sim.TileForm() in (other, ROWS)  # wide tiles against tuned rows on dense fluid: either
    sim.SetLanes([8] * len(V.TUNED_KERNELS))
    sim.SetState(s["x"], s["v"])
    sim.Steps(1)
    assert sim.TileForm() == ROWS
