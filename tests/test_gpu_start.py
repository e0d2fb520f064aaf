"""A run's start, which stays on the device, and the legacy solver's state, packed and scattered
there: at block and warp edges, bit for bit, since nothing here rounds but the split of a
cell-relative position, which a fresh simulation makes alike."""
import numpy as np
import pytest

import vfd_gb300 as V
from vfd_gb300 import scenes, sph

pytestmark = pytest.mark.gpu


def scene(n, seed):
    s = scenes.small_dam_break(n_side=max(2, int(np.ceil(n ** (1 / 3)))), r=0.01, viscosity=0.02)
    rng = np.random.default_rng(seed)
    return dict(s, x=s["x"][:n], v=rng.normal(0, 0.2, (n, 3)).astype(np.float32))


def state(sim, k=0):
    return [np.array(a) for a in sim.GetState(k)]


@pytest.mark.parametrize("n", [1, 255, 257, 1500])
@pytest.mark.parametrize("relative", [False, True])
def test_reset_is_a_fresh_start(n, relative):
    s, t = scene(n, 1), scene(n, 2)

    def make(u):
        sim = V.scene_simulation(u)
        sim.SetPositionMode(relative)
        return sim
    sim = make(s)
    start = state(sim)
    np.testing.assert_array_equal(start[1], s["v"])
    if not relative:
        np.testing.assert_array_equal(start[0], s["x"])
    sim.Steps(2)
    after = state(sim)
    sim.Reset()
    for a, b in zip(start, state(sim)):
        np.testing.assert_array_equal(a, b)
    sim.Steps(2)
    for a, b in zip(after, state(sim)):
        np.testing.assert_array_equal(a, b)
    sim.Emit(s["x"][:1] + np.float32([0, 0.5, 0]))
    sim.Steps(1)
    sim.Reset()  # the layout shrinks back
    sim.Steps(2)
    for a, b in zip(after, state(sim)):
        np.testing.assert_array_equal(a, b)
    sim.SetFluidObjects(t["x"], t["v"])  # the same layout, another start
    fresh = make(t)
    sim.Steps(2)
    fresh.Steps(2)
    for a, b in zip(state(fresh), state(sim)):
        np.testing.assert_array_equal(a, b)


def test_batch_reset_after_one_scene_changed():
    sc = [scene(n, n) for n in (1, 300, 64, 1000)]
    maps = [[V.build_box_map(b["min"], b["max"], b["inverted"], b["padding"], b["resolution"], 0.01) for b in s["boxes"]]
            for s in sc]
    sim = V.batch_simulation(sc, maps)
    sim.Steps(1)
    sc[1] = dict(sc[1], v=-sc[1]["v"])
    sim.SetFluidObjects(sc[1]["x"], sc[1]["v"], scene=1)
    sim.Reset()
    for k, s in enumerate(sc):
        x, v = state(sim, k)[:2]
        np.testing.assert_array_equal(x, s["x"])
        np.testing.assert_array_equal(v, s["v"])


def test_cell_relative_start_outside_the_anchors_is_refused():
    s = scene(64, 3)
    far = s["x"].copy()
    far[0, 1] += 1024 * 0.04  # cells of edge h = 0.04, 511 of them to each side of the centre
    sim = V.scene_simulation(dict(s, x=far))
    sim.SetPositionMode(True)
    for _ in range(2):
        with pytest.raises(V.VFDError):
            sim.Reset()
    far[0, 1] -= 8 * 0.04
    sim.SetFluidObjects(far, s["v"])
    sim.Reset()
    np.testing.assert_allclose(state(sim)[0], far, rtol=0, atol=4e-6)  # one place of 41 m


@pytest.mark.parametrize("n", [1, 255, 257, 4097])
def test_legacy_state_round_trip(n):
    rng = np.random.default_rng(n)
    x = rng.uniform(-0.1, 0.1, (n, 3)).astype(np.float32)
    v = rng.normal(0, 0.1, (n, 3)).astype(np.float32)
    sim = sph.SPHSimulation(sph.make_sph_desc(), x)
    sim.SetVelocities(v)
    a = sim.GetState()
    np.testing.assert_array_equal(a[0], x)
    np.testing.assert_array_equal(a[1], v)
