"""Surfaces whose boxes of corners, or of a normal's points, span more than the cells that lanes walk
together: the triangles and normals of the per-point densities, and no more time than a fine grid."""
import time

import numpy as np
import pytest

from fluid_gb300 import pbf, scenes
from tests import test_gpu_surface_grid as grid

pytestmark = pytest.mark.gpu


# a block of corners is one step wide, a cell about h = 0.1; the line lies at 1.25 cells
@pytest.mark.parametrize("step", [0.1, 0.125, 0.1255, 0.2, 0.37, 0.8])
def test_triangles_on_both_sides_of_the_line(step):
    grid.test_triangles_follow_the_corner_densities((-0.1, -0.05, 0.0), (1.1, 1.0, 1.0), step, 700)


def test_normals_whose_points_lie_cells_apart():
    h = 0.001  # the differences are taken over 0.002
    prm = scenes.physical_params(h, h / 2, box_lo=(0.0, 0.0, 0.0), box_hi=(0.02, 0.02, 0.02))
    pos = 0.005 + 0.008 * np.random.default_rng(0).uniform(0, 1, (3000, 3))
    with pbf.Simulator(pos, np.zeros_like(pos), prm) as sim:
        xyz, nrm = sim.surface(iso=0.3 * prm.rest_density, step=0.4 * h, lo=(0.0,) * 3, hi=(0.02,) * 3)
        assert len(xyz) > 100
        p, n = xyz.reshape(-1, 3), nrm.reshape(-1, 3)
        d = np.empty((2, 3, len(p)))
        for a in range(3):
            for k, sgn in enumerate((-1, 1)):
                q = p.copy()
                q[:, a] += np.float32(sgn * 0.001)
                d[k, a] = sim.estimate_density_at(q)
    g = (d[0] - d[1]).T
    length = np.linalg.norm(g, axis=1)
    # densities to 1e-6, the vertex to a few of its FP32 spacings (1e-6 of h) times the kernel's slope
    bound = 3e-5 * d.max() / np.maximum(length, 1e-30)
    ok = bound < 0.05
    assert ok.mean() > 0.9
    err = np.linalg.norm(n - g / np.maximum(length, 1e-30)[:, None], axis=1)
    assert (err[ok] <= bound[ok]).all()


def test_coarse_grids_cost_no_more_than_fine_ones():
    h = 0.02
    pos = np.random.default_rng(0).uniform(0.01, 0.99, (200000, 3))
    with pbf.Simulator(pos, np.zeros_like(pos), scenes.physical_params(h, h / 2)) as sim:
        def best(step):
            t = []
            for _ in range(6):
                t0 = time.perf_counter()
                sim.surface(step=step, lo=(0.0,) * 3, hi=(1.0,) * 3)
                t.append(time.perf_counter() - t0)
            return min(t)
        fine = best(h)
        for step in (4 * h, 16 * h, 0.5):
            assert best(step) < 2.0 * fine
