"""Surfaces whose cubes fill more tiles than one round of the tiles' scan (4,096 tiles of 2,048 cubes):
the triangles behind the first round are those of a box around them alone."""
import numpy as np
import pytest

from fluid_gb300 import pbf, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cubes", [203, 204, 210])  # 4,085, 4,146 and 4,522 tiles
def test_triangles_behind_the_first_round(cubes):
    step = 1.0 / 256.0  # corners at exact coordinates, the same in every box
    h = 8 * step
    prm = scenes.physical_params(h, h / 2, max_neighbors=256)
    end = (cubes - 1) * step
    pos = np.random.default_rng(0).uniform([end - 0.06, 0.3, 0.2], [end, 0.5, 0.7], (2000, 3))
    iso = 0.1 * prm.rest_density
    with pbf.Simulator(pos, np.zeros_like(pos), prm) as sim:
        near, near_n = sim.surface(iso=iso, step=step, lo=(end - 32 * step, 0.0, 0.0), hi=(end,) * 3)
        xyz, nrm = sim.surface(iso=iso, step=step, lo=(0.0,) * 3, hi=(end,) * 3)
    assert len(near) > 1000
    np.testing.assert_array_equal(xyz, near)
    np.testing.assert_array_equal(nrm, near_n)
