"""Batched scenes from a particle in two cells to forty a cell: windows walked by the whole warp or by its groups, on both sides of the
line (16 particles a stencil). A scene is as the single-scene solver has it, and bitwise itself whichever slots its
particles and their windows are in (other sort periods, other company)."""
import numpy as np
import pytest

from conftest import state_errors
from test_gpu_batch import _as_ref, _equal, _mixed_scenes
from test_gpu_parity import TARGET, _check

pytestmark = pytest.mark.gpu


def _scene(per_cell, seed):
    base = _mixed_scenes(k=3, steps=60)[1]
    rng = np.random.default_rng(seed)
    side = 24.0
    n = int(side * side * per_cell) + seed
    pos = np.array([20.0, base.border_margin + 0.4]) + side * rng.random((n, 2))
    pos[: n // 8] = pos[0]  # a heap in one stencil
    pos[: n // 8] += 0.3 * rng.random((n // 8, 2))
    vel = np.stack([-(pos[:, 1] - 15.0), pos[:, 0] - 32.0], 1) * 0.01 / base.delta_time / 24.0
    vol = np.full(n, 1.0 / per_cell, np.float32)
    return base.with_(position=pos.astype(np.float32), velocity=vel.astype(np.float32), volume=vol,
                      mass=vol * np.float32(base.rho / 100.0))


@pytest.mark.parametrize("per_cell", [0.5, 1, 4, 15, 17, 40])
def test_density(gpu_lib, per_cell):
    from mpm_snow_sim2d_b200 import Solver
    from mpm_snow_sim2d_b200.batch import Batch
    scs = [_scene(per_cell, s) for s in (1, 2)]

    def run(order, period):
        with Batch([scs[i] for i in order]) as b:
            b.set_config(sort_period=period)
            b.step(30)
            return {i: (b.get_state(j), b.status(j)) for j, i in enumerate(order)}

    a, b = run([0, 1], 16), run([1, 0], 1)
    for i in range(2):
        assert a[i][1] == b[i][1] and a[i][1] & 3 == 0
        assert _equal(a[i][0], b[i][0]), i
        with Solver.from_scene(scs[i]) as s:
            s.Step(30)
            _check(state_errors(a[i][0], _as_ref(s.get_state()), 2), TARGET, f"scene {i} vs single-scene solver")
