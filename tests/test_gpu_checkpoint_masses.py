"""Checkpoints of solvers whose particles have masses and volumes of their own: the run goes on bitwise, in a new solver and in one
that has sorted its particles another way since."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("masses,volumes", [(True, True), (True, False), (False, True)])
def test_resume(gpu_lib, tmp_path, dim, masses, volumes):
    from mpm_snow_sim2d_b200 import Solver, scenes
    sc = scenes.impact_3d(steps=64) if dim == 3 else scenes.impact_2d(steps=64)
    rng = np.random.default_rng(dim)
    mass = sc.mass * (rng.uniform(0.7, 1.3, sc.count).astype(np.float32) if masses else np.float32(1))
    volume = sc.volume * (rng.uniform(0.7, 1.3, sc.count).astype(np.float32) if volumes else np.float32(1))
    sc = sc.with_(mass=mass.astype(np.float32), volume=volume.astype(np.float32))
    fields = ("position", "velocity", "affine_b", "elastic_f", "plastic_det")
    path = tmp_path / "state"
    with Solver.from_scene(sc) as s:
        s.Step(7)
        s.save(path)
        s.Step(40)
        want = s.get_state()
        s.load(path)  # from another slot order
        s.Step(40)
        again = s.get_state()
    with Solver.from_scene(sc) as s:
        s.load(path)
        s.Step(40)
        got = s.get_state()
    for f in fields:
        assert np.array_equal(getattr(got, f), getattr(want, f)), f
        assert np.array_equal(getattr(again, f), getattr(want, f)), f
