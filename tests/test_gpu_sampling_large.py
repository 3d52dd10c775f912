"""The sampler where a phase's cells change from eight lanes to one: grids whose phases lie on both sides of the line, bit for bit as the
numpy restatement has them."""
import numpy as np
import pytest

from oracle import sample_ref
from test_gpu_sampling import _shape

pytestmark = pytest.mark.gpu


# 2D: 304 cells a side, phases of 10201 to 10404 cells (line: 10240); 3D: 88 a side, 24389 to 27000 (24576)
@pytest.mark.parametrize("dim,side,rounds", [(2, 304, 5), (3, 88, 2)])
def test_phases_on_both_sides(gpu_lib, dim, side, rounds):
    from mpm_snow_sim2d_b200.sampling import sample_shapes
    cell = 1.0 / np.sqrt(dim)
    half = (0.5 * cell * (side - 1.5),) * dim
    c = (0.21,) * dim
    shapes = [_shape(1, c, h=half + (0.0,) * (3 - dim)), _shape(0, c, half[0] / 2)]
    got, owner = sample_shapes(dim, shapes, 1.0, 7, rounds)
    ref, ref_owner = sample_ref.sample_shapes(dim, shapes, 1.0, 7, rounds)
    assert got.shape == ref.shape and got.shape[0] > 10000
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32)) and np.array_equal(owner, ref_owner)
