"""The FP64 path at the sizes where its lanes per particle change (8 below 4,000 particles, 4
below 12,000, 2 below 100,000, then 1) and after a reset, against the FP64 CPU oracle: the
iteration counts and the 1e-9 h of test_gpu_fp64.py (double rounding times a few hundred
operations in a row, 1e-13 of the position, leaves four decimal places of room)."""
import numpy as np
import pytest

from vfd_gb300 import scenes
from test_gpu_fp64 import run_and_compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3999, 4000, 11999, 12000, 99999, 100001])
def test_lane_counts(n):
    s = scenes.small_dam_break(n_side=max(2, int(np.ceil(n ** (1 / 3)))), r=0.01, viscosity=0.02, surface_tension=0.05)
    x = s["x"][:n]
    v = np.stack([np.sin(9 * x[:, 1]), np.cos(7 * x[:, 2]), np.sin(8 * x[:, 0])], 1).astype(np.float32) if n > 1 else 0 * x
    s = dict(s, x=x, v=v)
    s["desc"] = dict(s["desc"], MaxDivergenceSolverIterations=7)
    g = run_and_compare(s, 2, 1e-9)
    first = g.GetStateF64()
    g.Reset()  # the buffers serve again: the same run
    g.Steps(2)
    for a, b in zip(first, g.GetStateF64()):
        np.testing.assert_array_equal(a, b)
