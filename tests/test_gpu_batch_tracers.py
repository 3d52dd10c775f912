"""Particles without volume add nothing to the grid and read it: where no mass is near, nothing moves them."""
import numpy as np
import pytest

from test_gpu_batch import _equal, _mixed_scenes

pytestmark = pytest.mark.gpu


def _scene(edge):
    """A block that moves off to the right, 0.25 cells a step, and tracers spread over where it was; with `edge` the same at the lower
    wall of the domain, some tracers with stencils that reach outside."""
    sc = _mixed_scenes(k=3, steps=200)[2]
    rng = np.random.default_rng(5)
    y0 = 0.0 if edge else 40.0
    n, m = 2000, 300
    body = np.stack([30 + 16 * rng.random(n), y0 + 3 + 10 * rng.random(n)], 1)
    tracers = np.stack([28 + 20 * rng.random(m), y0 + 0.2 + 14 * rng.random(m)], 1)
    vel = np.zeros((n + m, 2), np.float32)
    vel[:n, 0] = 0.25 / sc.delta_time
    vol = np.full(n + m, sc.volume[0], np.float32)
    vol[n:] = 0.0
    return sc.with_(position=np.concatenate([body, tracers]).astype(np.float32), velocity=vel, volume=vol,
                    mass=np.full(n + m, sc.mass[0], np.float32), gravity=0.0), n


@pytest.mark.parametrize("edge", [False, True])
def test_tracers_left_behind_stand_still(gpu_lib, edge):
    from mpm_snow_sim2d_b200.batch import Batch
    sc, n = _scene(edge)
    with Batch([sc]) as b:
        b.step(160)
        st = b.get_state(0)
    body, tr = st.position[:n], st.position[n:]
    near = np.array([np.any(np.all(np.abs(body - p) < 5.0, axis=1)) for p in tr])
    assert (~near).sum() > 50
    assert np.all(st.velocity[n:][~near] == 0.0)


def test_tracers_do_not_depend_on_company(gpu_lib):
    from mpm_snow_sim2d_b200.batch import Batch
    scs = [_scene(False)[0], _scene(True)[0]] + _mixed_scenes(k=2, steps=200)
    with Batch(scs) as b:
        b.step(100)
        b.step(37)
        got = [b.get_state(k) for k in range(2)]
    for k in range(2):
        with Batch([scs[k]]) as b:
            b.set_config(sort_period=7)
            b.step(137)
            assert _equal(b.get_state(0), got[k]), k
