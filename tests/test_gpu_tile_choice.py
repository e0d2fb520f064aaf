"""Each step takes the form of the staged tiles that is cheapest for its own state, however the state
came about (set, restored, queued, launched by the host) and whatever ran before it: narrow tiles on a
lattice, rows on sparse fluid and where halos outgrow the shared memory, wide tiles on denser fluid from
700,000 particles on. The states here lie well inside the range of each form (by the steps that the
rule is fitted to, its choice is 10 % faster than the next, or 3 % where the note says so)."""
import numpy as np
import pytest

from test_gpu_halo import block_scene
import vfd_gb300 as V

pytestmark = pytest.mark.gpu

SMALL, LARGE = (69, 69, 69), (89, 90, 91)  # 328,509 and 728,910 particles
ROWS, NARROW, WIDE = 0, 1, 2


def scene(counts, squeeze=1.0, keep=1.0):
    """A lattice at rest; squeezed to 0.95 of the spacing its tiles outgrow the narrow form, at 0.88 the wide one."""
    s = block_scene(counts, 0.05)
    x = s["x"] * np.float32(squeeze)
    if keep < 1:
        x = x[np.random.default_rng(2).random(len(x)) < keep]
    return dict(s, x=x, v=0 * x,
                desc=dict(s["desc"], MaxPressureSolverIterations=3, MaxDivergenceSolverIterations=3,
                          MaxViscositySolverIterations=3))


@pytest.mark.parametrize("counts,other", [(SMALL, ROWS), (LARGE, WIDE)])
def test_set_states(counts, other):
    s, dense = scene(counts), scene(counts, 0.95)
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


@pytest.mark.parametrize("counts,squeeze,keep", [
    ((47, 48, 49), 1.0, 1.0),   # 110,544 particles: few more tiles than blocks run at once
    (LARGE, 1.0, 0.3),          # 70 particles a tile
    (LARGE, 0.88, 1.0)])        # halos beyond the shared memory of either form
def test_states_that_rows_suit(counts, squeeze, keep):
    sim = V.scene_simulation(scene(counts, squeeze, keep))
    sim.Steps(1)
    assert sim.TileForm() == ROWS


def test_batch_of_small_scenes():
    s = block_scene((8, 8, 8), 0.0)  # 200 scenes of 512 particles: 64 a tile
    sim = V.DFSPHSimulation(scenes=[V._abi.make_desc(**s["desc"])] * 200)
    for k in range(200):
        sim.SetFluidObjects(s["x"], 0 * s["v"], scene=k)
    sim.Steps(1)
    assert sim.TileForm() == ROWS


@pytest.mark.parametrize("counts,other", [(SMALL, ROWS), (LARGE, WIDE)])
@pytest.mark.parametrize("tuned_on_lattice", [True, False])
def test_tuning_keeps_the_forms_it_does_not_find_slower(counts, other, tuned_on_lattice):
    s, dense = scene(counts), scene(counts, 0.95)
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
    assert sim.TileForm() in (other, ROWS)  # (wide tiles against tuned rows: either)
    sim.SetLanes([8] * len(V.TUNED_KERNELS))
    sim.SetState(s["x"], s["v"])
    sim.Steps(1)
    assert sim.TileForm() == ROWS
    sim.SetTileForm(WIDE)
    sim.Steps(1)
    assert sim.TileForm() == WIDE
    sim.SetTileForm()
    sim.SetState(s["x"], s["v"])
    sim.Steps(1)
    assert sim.TileForm() == NARROW
