"""The grid sums of the split transfer (MPM_TRANSFER=split), which lie channel by channel: mass and momentum of the particles, the raw
sums in the order the interface states, and those of the fused transfer for the same state within the rounding of its windows."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("quadratic", [False, True])
def test_sums(gpu_lib, dim, quadratic):
    from mpm_snow_sim2d_b200 import Solver, _lib, scenes
    sc = scenes.impact_3d() if dim == 3 else scenes.impact_2d()
    if quadratic:
        sc = sc.with_(formulation=_lib.FORMULATION_MLS_QUADRATIC)
    out = {}
    for transfer in ("split", "fused"):
        old = os.environ.get("MPM_TRANSFER")
        os.environ["MPM_TRANSFER"] = transfer
        try:
            with Solver.from_scene(sc) as s:
                mass, mom, raw = s.rasterize(raw=True)
                lm, lp = s.fixed_point()[:2]
                s.Step(3)
                out[transfer] = (mass, mom, raw, s.rasterize()[0], s.get_state())
        finally:
            os.environ.pop("MPM_TRANSFER") if old is None else os.environ.update(MPM_TRANSFER=old)
        raw = np.asarray(raw).reshape(1 + dim, -1)
        assert np.array_equal(raw[0] * 2.0 ** -lm, np.ravel(mass))
        assert np.array_equal((raw[1:] * 2.0 ** -lp).T.ravel(), np.ravel(mom))
    a, b = out["split"], out["fused"]
    total = float(sc.mass.astype(np.float64).sum())
    for k in (0, 3):
        assert abs(a[k].sum() - total) <= 1e-6 * total
        assert np.linalg.norm(a[k] - b[k]) <= 1e-6 * np.linalg.norm(b[k])
    assert np.linalg.norm(a[1] - b[1]) <= 1e-6 * np.linalg.norm(b[1])


@pytest.mark.parametrize("width,height", [(2047, 2047), (2600, 1700)])  # just 4 Mi nodes, and some more
def test_sums_of_large_grids(gpu_lib, width, height):
    from mpm_snow_sim2d_b200 import Solver, scenes
    sc = scenes.impact_2d().with_(width=width, height=height)
    rng = np.random.default_rng(width)
    n = 3000
    pos = np.array([3.0, 3.0]) + rng.random((n, 2)) * (np.array([width, height]) - 6.0)
    sc = sc.with_(position=pos.astype(np.float32), velocity=rng.standard_normal((n, 2)).astype(np.float32),
                  volume=np.full(n, sc.volume[0], np.float32), mass=np.full(n, sc.mass[0], np.float32))
    with Solver.from_scene(sc) as s:
        mass, mom, raw = s.rasterize(raw=True)
        lm, lp = s.fixed_point()[:2]
    nodes = (width + 1) * (height + 1)
    assert np.array_equal(raw.reshape(3, nodes)[0] * 2.0 ** -lm, mass)
    assert np.array_equal(raw.reshape(3, nodes)[1:].T * 2.0 ** -lp, mom)
    x = np.floor(pos.astype(np.float32)).astype(np.int64)
    near = np.zeros((height + 1, width + 1), bool)  # the nodes of every stencil, and no others
    for a in range(-1, 3):
        for b in range(-1, 3):
            near[x[:, 1] + b, x[:, 0] + a] = True
    got = mass.reshape(height + 1, width + 1)
    assert np.all(got[~near] == 0) and abs(got.sum() - sc.mass.astype(np.float64).sum()) <= 1e-5 * got.sum()
