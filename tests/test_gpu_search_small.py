"""The one-launch search of small scenes against the oracle, bit for bit: particle counts at and
beside a block, a round of the cluster and the largest it takes (above it the general search
runs), tables whose cells are not a multiple of the cluster's threads, everything in one cell,
non-finite positions and a table that has to grow."""
import numpy as np
import pytest

import vfd_gb300 as V
from oracle import oracle as O
from vfd_gb300 import scenes
from test_gpu_parity import assert_neighbors_equal

pytestmark = pytest.mark.gpu


def scene(n, side):
    s = scenes.small_dam_break(n_side=8)
    h = 4 * s["desc"]["ParticleRadius"]
    x = (side * h * np.random.default_rng(n).random((n, 3))).astype(np.float32)
    return dict(s, x=x, v=np.zeros_like(x), boxes=[])


def check(sim, s):
    o = O.scene_oracle(s, 32, maps=[])
    sim.FindNeighbors()
    o.find_neighbors()
    assert_neighbors_equal(sim, o)


@pytest.mark.parametrize("n,side", [
    (1, 1.0), (31, 0.9), (1023, 3.0), (1025, 40.0), (8191, 9.0), (8193, 9.0), (16385, 61.0),
    (32768, 14.0), (32769, 14.0)])
def test_search_matches_oracle(n, side):
    s = scene(n, side)
    check(V.scene_simulation(s), s)


def test_table_grows_and_bad_positions_are_refused():
    s = scene(4000, 6.0)
    sim = V.scene_simulation(s)
    check(sim, s)
    far = s["x"].copy()
    far[7] += 3.0
    sim.SetState(far, s["v"])  # more cells than the table was sized for
    check(sim, dict(s, x=far))
    with pytest.raises(V.VFDError):
        sim.SetState(np.full_like(far, np.inf), s["v"])
    sim.SetState(s["x"], s["v"])
    check(sim, s)
