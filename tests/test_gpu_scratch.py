"""Reads, uploads and pictures borrow the buffers that a sort writes: they allocate no device memory, and what they leave there
changes no later step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _solver(dim):
    from mpm_snow_sim2d_b200 import Solver, scenes
    sc = scenes.impact_3d(steps=64) if dim == 3 else scenes.impact_2d(steps=64)
    reps = -(-60000 // sc.count)  # a field of every kind is then larger than the pieces that allocations are cut from
    rng = np.random.default_rng(dim)
    jit = lambda a: np.concatenate([a + rng.uniform(-0.2, 0.2, a.shape) for _ in range(reps)]).astype(np.float32)  # noqa: E731
    return Solver.from_scene(sc.with_(position=jit(sc.position), velocity=np.tile(sc.velocity, (reps, 1)),
                                      volume=np.tile(sc.volume, reps) / reps, mass=np.tile(sc.mass, reps) / reps))


@pytest.mark.parametrize("dim", [2, 3])
def test_first_calls_allocate_nothing(gpu_lib, dim):
    with _solver(dim) as other:  # what the process makes once
        other.Step(1)
        other.GetParticlePositions()
        st = other.get_state()
        other.render(width=64, height=64, point_size=1.0)
        other.set_state(st.position, st.velocity, st.affine_b, st.elastic_f, st.plastic_det)
    with _solver(dim) as s:
        s.Step(1)
        free = _free()
        s.GetParticlePositions()
        st = s.get_state()
        s.render(width=300, height=200, point_size=1.0)
        s.set_state(st.position, st.velocity, st.affine_b, st.elastic_f, st.plastic_det)
        assert _free() == free


def test_first_calls_of_a_batch_allocate_nothing(gpu_lib):
    from mpm_snow_sim2d_b200 import scenes
    from mpm_snow_sim2d_b200.batch import Batch
    sc = scenes.batch_scene_2d(3)
    rng = np.random.default_rng(0)
    n = 200000
    sc = sc.with_(position=(sc.width * rng.uniform(0.2, 0.8, (n, 2))).astype(np.float32), velocity=np.zeros((n, 2), np.float32),
                  volume=np.full(n, sc.volume[0] / 50, np.float32), mass=np.full(n, sc.mass[0] / 50, np.float32))
    with Batch([scenes.batch_scene_2d(5)]) as other:
        other.step(1)
        st = other.get_state(0)
        other.set_state(0, st.position, st.velocity)
    with Batch([sc]) as b:
        b.step(1)
        free = _free()
        st = b.get_state(0)
        b.set_state(0, st.position, st.velocity)
        assert _free() == free


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("steps", [1, 5])
def test_reading_between_steps_changes_nothing(gpu_lib, dim, steps):
    """Over several sorts, with and without reads in between: the same run, bitwise."""
    def run(read):
        with _solver(dim) as s:
            for _ in range(60 // steps):
                s.Step(steps)
                if read:
                    s.render(width=320, height=240, point_size=2.0)
                    s.get_state()
                    s.GetParticlePositions()
            st = s.get_state()
            return [st.position, st.velocity, st.affine_b, st.elastic_f, st.plastic_det]
    assert all(np.array_equal(a, b) for a, b in zip(run(True), run(False)))


def test_picture_larger_than_the_buffers(gpu_lib):
    """A tiny solver's picture takes memory of its own: the same picture as the next one."""
    from mpm_snow_sim2d_b200 import Solver, scenes
    sc = scenes.impact_2d(steps=4)
    sc = sc.with_(position=sc.position[:50], velocity=sc.velocity[:50], volume=sc.volume[:50], mass=sc.mass[:50])
    with Solver.from_scene(sc) as s:
        a = s.render(width=700, height=500, point_size=3.0)
        s.get_state()
        assert np.array_equal(a, s.render(width=700, height=500, point_size=3.0)) and a.any()
