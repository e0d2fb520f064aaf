"""States set from and read into pinned, pageable and mixed host arrays, at addresses that are not a
float's, and non-finite values in each: the same bytes and the same refusals whichever way the
arrays travel."""
import ctypes as C

import numpy as np
import pytest

import vfd_gb300 as V
from vfd_gb300 import scenes

pytestmark = pytest.mark.gpu

N = 1331


def pinned(a, shift=0):
    """The array in pinned memory, `shift` bytes into an allocation with room behind it."""
    import torch
    raw = torch.zeros(a.nbytes + 64, dtype=torch.uint8, pin_memory=True).numpy()
    out = raw[shift:shift + a.nbytes].view()
    out[:] = np.ascontiguousarray(a).view(np.uint8).reshape(-1)
    return out


def pageable(a):
    return np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()


def ptr(a):
    return C.cast(C.c_void_p(a.ctypes.data), C.POINTER(C.c_float)) if a is not None else None


def set_state(sim, x, v):
    return V.lib().vfd_set_state(sim._h, ptr(x), ptr(v))  # the arrays live until it returns


def make():
    sim = V.scene_simulation(scenes.small_dam_break(n_side=11, r=0.01))
    x, v, _ = sim.GetState()
    assert len(x) == N
    rng = np.random.default_rng(1)
    return sim, x + np.float32(1e-3) * rng.random((N, 3), np.float32), rng.normal(0, 0.1, (N, 3)).astype(np.float32)


@pytest.mark.parametrize("px,pv", [(0, 0), (4, 0), (0, None), (None, 0), (None, None), (1, 0), (0, 2), (3, 3)])
def test_set_and_read(px, pv):
    sim, x, v = make()
    place = lambda a, s: pageable(a) if s is None else pinned(a, s)  # noqa: E731
    assert set_state(sim, place(x, px), place(v, pv)) == 0
    for a, b in zip(sim.GetState(), (x, v)):
        np.testing.assert_array_equal(a, b)
    out = [place(np.zeros_like(x), s) for s in (px, pv, px)]
    assert V.lib().vfd_scene_get_state(sim._h, 0, *(ptr(o) for o in out)) == 0
    for a, b in zip(out, sim.GetState()):
        np.testing.assert_array_equal(a, b.view(np.uint8).reshape(-1))
    one = place(np.zeros_like(x), px)
    assert V.lib().vfd_scene_get_state(sim._h, 0, None, ptr(one), None) == 0
    np.testing.assert_array_equal(one, v.view(np.uint8).reshape(-1))


@pytest.mark.parametrize("place", [lambda a: pinned(a), lambda a: pinned(a, 1), pageable])
@pytest.mark.parametrize("which,at", [(0, 0), (1, 3 * N - 1)])
def test_non_finite_values_are_refused(place, which, at):
    sim, x, v = make()
    before = sim.GetState()
    bad = [x.copy(), v.copy()]
    bad[which].reshape(-1)[at] = np.nan
    assert set_state(sim, *(place(a) for a in bad)) != 0
    for a, b in zip(before, sim.GetState()):
        np.testing.assert_array_equal(a, b)
    assert set_state(sim, place(x), place(v)) == 0  # the refusal does not stay
    np.testing.assert_array_equal(sim.GetState()[0], x)
