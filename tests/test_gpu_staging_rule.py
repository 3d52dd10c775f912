"""Scenes around the line between gathered and staged node boxes (windows per warp, particles per cell), as the solver runs them by
itself against the other kernel forced on them: the same windows, so equal but for how the two builds contract multiply-adds."""
import os

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _scene(dim, n, per_cell, quadratic):
    """n particles over a ragged grid down to its walls, falling and spinning."""
    from mpm_snow_sim2d_b200 import _lib, scenes
    base = scenes.impact_3d() if dim == 3 else scenes.impact_2d()
    rng = np.random.default_rng(n)
    side = (n / per_cell) ** (1.0 / dim)
    ext = [int(side * f) + 9 for f in (1.3, 1.1, 1.0)][:dim]
    pos = base.border_margin + 0.3 + rng.random((n, dim)) * side
    vel = np.zeros((n, dim))
    vel[:, 0], vel[:, 1] = -(pos[:, 1] - ext[1] / 2), pos[:, 0] - ext[0] / 2
    vel *= 0.02 / base.delta_time / max(ext)
    form = _lib.FORMULATION_MLS_QUADRATIC if quadratic else _lib.FORMULATION_MLS
    vol = np.full(n, 1.0 / per_cell, np.float32)
    return base.with_(width=ext[0], height=ext[1], depth=ext[2] if dim == 3 else 0, position=pos.astype(np.float32),
                      velocity=vel.astype(np.float32), volume=vol, mass=(vol * np.float32(base.rho / 100.0)), formulation=form)


# windows per warp (of 2960) above and below each line, particles per cell above and below
@pytest.mark.parametrize("dim,n,per_cell,quadratic,other", [
    (2, 1500007, 8, False, "gather"), (2, 1500007, 4, True, "gather"), (2, 1200007, 8, False, "tma"), (2, 1500007, 3, False, "tma"),
    (3, 320007, 8, False, "gather"), (3, 320007, 3, False, "gather"), (3, 320007, 2, False, "tma"), (3, 250007, 8, False, "tma"),
    (3, 1600007, 8, True, "gather"), (3, 1600007, 4, True, "tma")])
def test_either_side(gpu_lib, dim, n, per_cell, quadratic, other):
    from mpm_snow_sim2d_b200 import Solver
    sc = _scene(dim, n, per_cell, quadratic)

    def run(force):
        old = os.environ.pop("MPM_BOX_LOAD", None)
        try:
            if force:
                os.environ["MPM_BOX_LOAD"] = force
            with Solver.from_scene(sc) as s:
                s.Step(12)
                return s.get_state(), s.status()
        finally:
            os.environ.pop("MPM_BOX_LOAD", None)
            if old is not None:
                os.environ["MPM_BOX_LOAD"] = old

    (a, fa), (b, fb) = run(None), run(other)
    assert fa == fb and fa & (1 | 2 | 16) == 0
    # twelve steps, a few roundings of 2^-24 each; the bounds of the longer runs of test_gpu_fused.py
    for f, bound in (("position", 1e-6), ("elastic_f", 1e-5), ("plastic_det", 1e-5)):
        assert rel_l2(getattr(a, f), getattr(b, f)) < bound, f
