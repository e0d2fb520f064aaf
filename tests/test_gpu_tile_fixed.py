"""The passes of either form of the staged tiles, fixed whatever the state would choose, against the
FP32 oracle and the row kernels: the scenes and bounds of test_gpu_halo.py (ragged blocks, halos that
outgrow the shared memory, tiles of a single particle, uneven batches), the analytic kernel, and the
adjoint's recorded steps."""
import numpy as np
import pytest

import test_gpu_halo as H
import vfd_gb300 as V
from vfd_gb300 import _abi

pytestmark = pytest.mark.gpu

FORMS = pytest.mark.parametrize("form", [1, 2])


def on_form(monkeypatch, form):
    """Simulations made by the scenes' helpers run on `form` (until lanes are set)."""
    for name in ("scene_simulation", "batch_simulation"):
        def make(*a, _make=getattr(V, name), **k):
            sim = _make(*a, **k)
            sim.SetTileForm(form)
            return sim
        monkeypatch.setattr(V, name, make)


@FORMS
@pytest.mark.parametrize("counts,tension,relative", [((47, 48, 49), 0.0, False), ((50, 41, 53), 0.05, True)])
def test_step_matches_oracle(monkeypatch, form, counts, tension, relative):
    on_form(monkeypatch, form)
    H.test_step_matches_oracle(counts, tension, relative)


@FORMS
@pytest.mark.parametrize("relative", [False, True])
def test_crowded_halos_and_lone_particles(monkeypatch, form, relative):
    on_form(monkeypatch, form)
    H.test_crowded_halos_and_lone_particles(relative)


@FORMS
def test_batch_of_uneven_scenes(monkeypatch, form):
    on_form(monkeypatch, form)
    H.test_batch_of_uneven_scenes()


@FORMS
@pytest.mark.parametrize("squeeze", [1.0, 0.88])
def test_analytic_kernel(form, squeeze):
    s = H.block_scene((47, 48, 49), 0.05)
    s = dict(s, x=s["x"] * np.float32(squeeze), desc=dict(s["desc"], MaxPressureSolverIterations=5,
                                                          MaxDivergenceSolverIterations=5, MaxViscositySolverIterations=5))

    def make():
        sim = V.scene_simulation(s)
        sim.SetKernelMode(True)
        sim.SetTileForm(form)
        return sim
    H.assert_like_rows(make)


@pytest.mark.parametrize("counts,form,squeeze", [
    ((47, 47, 47), 1, 1.0), ((47, 47, 47), 2, 1.0), ((64, 64, 64), -1, 1.0), ((47, 47, 47), -1, 0.9)])
@pytest.mark.parametrize("graphs", [True, False])
def test_recorded_steps(counts, form, squeeze, graphs):
    """Gradients of two recorded steps and their replay, on the analytic kernel with a fixed step length, on a fixed
    form and on the one that the steps choose (narrow tiles; rows): the recorded states agree with the
    rows' to 1e-6 (test_gpu_halo.py), and a gradient is a smooth function of them here, so a bound of
    1e-4 of its norm leaves a factor of a hundred."""
    s = H.block_scene(counts, 0.0)
    s = dict(s, x=s["x"] * np.float32(squeeze),
             desc=dict(s["desc"], MaxTimeStepSize=1e-4, TimeStepSize=1e-4, MaxPressureSolverIterations=5,
                       MaxDivergenceSolverIterations=5, MaxViscositySolverIterations=5))
    rng = np.random.default_rng(4)
    bars = [rng.normal(0, 1, s["x"].shape).astype(np.float32) / len(s["x"]) for _ in range(2)]
    got = []
    for f in (form, 0):
        sim = V.scene_simulation(s)
        sim.SetKernelMode(True)
        sim.SetGraphMode(graphs)
        sim.SetTileForm(f)
        sim.AdjointForward(2, 1)
        got.append(sim.GetState()[:2] + tuple(sim.AdjointBackward(*bars)[:2]))
        assert sim.GetGraphMode() == (graphs, graphs)
    for a, b in zip(*got):
        assert np.isfinite(a).all()
        assert np.linalg.norm(a - b) <= 1e-4 * np.linalg.norm(b)


def test_forms_are_checked_and_small_layouts_run_rows():
    sim = V.scene_simulation(H.block_scene((9, 9, 9), 0.0))
    for bad in (-2, 3):
        with pytest.raises(V.VFDError):
            sim.SetTileForm(bad)
    sim.SetTileForm(1)
    sim.Steps(1)
    assert sim.TileForm() == 0 and sim.GetField(_abi.FIELD_DENSITY).min() > 0
