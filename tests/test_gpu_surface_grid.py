"""The surface's field passes where their blocks and shortcuts end: grids with remainders in every
axis, corners outside the particles' grid, particles at the box's walls, few particles. The field's
sign decides the triangles, so the triangle list is compared with one made from the density at the
corners (pbf_estimate_density_at), cube by cube."""
import numpy as np
import pytest

from fluid_gb300 import pbf, scenes

pytestmark = pytest.mark.gpu

CORNER = np.array([[0, 0, 0], [0, 1, 0], [1, 1, 0], [1, 0, 0], [0, 0, 1], [0, 1, 1], [1, 1, 1], [1, 0, 1]])


def _axis(lo, hi, step):
    nc = int(np.floor((hi - lo) / step)) + 1
    return np.minimum(lo + np.arange(nc + 1) * step, hi).astype(np.float32)


@pytest.mark.parametrize("lo,hi,step", [
    ((0.0, 0.0, 0.0), (1.0, 1.0, 1.0), 0.0499),
    ((-0.3, -0.2, -0.25), (1.2, 1.31, 1.17), 0.067),   # corners far outside the grid
    ((0.1, 0.0, 0.2), (0.47, 0.03, 0.9), 0.031),       # one cube thick
    ((0.4, 0.4, 0.4), (0.4, 0.4, 0.4), 0.1),           # a single corner
])
@pytest.mark.parametrize("n", [1, 700])
def test_triangles_follow_the_corner_densities(lo, hi, step, n):
    h = 0.1
    prm = scenes.physical_params(h, h / 2)
    rng = np.random.default_rng(n)
    pos = rng.uniform(0.0, 1.0, (n, 3)) * [0.5, 0.4, 1.0]
    pos[: n // 8, 0] = 0.0  # on a wall
    iso = 0.3 * prm.rest_density if n > 1 else 0.1 * prm.rest_density
    ax = [_axis(lo[a], hi[a], step) for a in range(3)]
    grid = np.stack(np.meshgrid(*ax, indexing="ij"), -1)
    edges, ntri, tri = pbf.mc_table()
    with pbf.Simulator(pos, np.zeros_like(pos), prm) as sim:
        xyz, nrm = sim.surface(iso=iso, step=step, lo=lo, hi=hi)
        dens = sim.estimate_density_at(grid.reshape(-1, 3)).reshape(grid.shape[:3])
    nc = [len(a) - 1 for a in ax]
    below = dens < np.float32(iso)
    want = []
    for ix in range(nc[0]):
        for iy in range(nc[1]):
            for iz in range(nc[2]):
                ci = sum(1 << k for k, c in enumerate(CORNER) if below[ix + c[0], iy + c[1], iz + c[2]])
                want += [(ix, iy, iz)] * int(ntri[ci])
    assert len(xyz) == len(want)
    for t, (ix, iy, iz) in enumerate(want):  # every triangle in its cube
        for a, k in enumerate((ix, iy, iz)):
            assert xyz[t, :, a].min() >= ax[a][k] - 1e-6 and xyz[t, :, a].max() <= ax[a][k + 1] + 1e-6
    if len(want):
        assert np.isfinite(nrm).all()
