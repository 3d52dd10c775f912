"""Contributions to a batched scene's grid that are not numbers or do not fit: flagged in the scene that makes them, counted as
0 (not a number), and without effect on the other scenes."""
import numpy as np
import pytest

from test_gpu_batch import _equal, _mixed_scenes

pytestmark = pytest.mark.gpu

NAN_STATE, OVERFLOW, OUTSIDE = 1, 2, 4


def _edge(sc, inside):
    """Two particles (their contributions to a node would cancel in 64 bits): in the middle, or in the domain's corner, where
    part of the stencil lies outside the grid."""
    at = [sc.width / 2, sc.height / 2] if inside else [0.4, 0.4]
    n = 2
    return sc.with_(position=np.tile(np.float32(at), (n, 1)), velocity=np.zeros((n, 2), np.float32),
                    volume=np.full(n, sc.volume[0], np.float32), mass=np.full(n, sc.mass[0], np.float32))


@pytest.mark.parametrize("inside", [True, False])
def test_stress_that_is_not_a_number(gpu_lib, inside):
    from mpm_snow_sim2d_b200.batch import Batch
    scs = _mixed_scenes(k=3, steps=20)
    bad = _edge(scs[1], inside).with_(youngs=float("nan"))
    with Batch([scs[0], bad, scs[2]]) as b:
        b.step(1)
        got, flags = [b.get_state(s) for s in range(3)], [b.status(s) for s in range(3)]
    with Batch([scs[0], scs[2]]) as b:
        b.step(1)
        ref, clean = [b.get_state(s) for s in range(2)], [b.status(s) for s in range(2)]
    assert flags[1] & NAN_STATE and not flags[1] & OVERFLOW
    assert bool(flags[1] & OUTSIDE) == (not inside)
    # their momentum counts as 0: gravity alone moves them
    assert np.isfinite(got[1].position).all() and np.isfinite(got[1].velocity).all()
    assert np.all(got[1].velocity[:, 0] == 0)
    assert [flags[0], flags[2]] == clean
    assert _equal(got[0], ref[0]) and _equal(got[2], ref[1])


@pytest.mark.parametrize("inside", [True, False])
def test_contribution_out_of_range(gpu_lib, inside):
    from mpm_snow_sim2d_b200.batch import Batch
    scs = _mixed_scenes(k=2, steps=20)
    with Batch([scs[0], _edge(scs[1], inside)]) as b:
        b.set_state(1, affine_b=np.full((2, 2, 2), 1e30, np.float32))
        b.step(1)
        flags = [b.status(s) for s in range(2)]
    assert flags[1] & OVERFLOW
    assert not flags[0] & (NAN_STATE | OVERFLOW)
