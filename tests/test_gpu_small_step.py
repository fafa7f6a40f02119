"""The whole-step kernel of small scenes against the per-phase kernels (which a profiled step
takes): the same bits in positions, velocities, densities, neighbour sets and statistics, at the
ends of its forms, for every option it is compiled for, and where its stages have remainders."""
import numpy as np
import pytest

from fluid_gb300 import pbf, scenes
from fluid_gb300.params import PBF_FLAG_GRAPH, PBF_FLAG_KEEP_PREDICTED, PBF_FLAG_STATS

pytestmark = pytest.mark.gpu

H = 0.05


def _state(n, jitter=0.2, seed=0):
    rng = np.random.default_rng(seed)
    s = min(H / 2, 0.9 / np.ceil(n ** (1 / 3)))
    side = int(np.ceil(n ** (1 / 3)))
    p = scenes.lattice(side, side, side, s, corner=(0.02, 0.0, 0.03))[:n]
    return p + rng.uniform(-jitter, jitter, p.shape) * s, rng.uniform(-1, 1, p.shape), 2 * s


def _run(pos, vel, prm, profiled, steps=2, counts=None):
    boxes = [(prm.box_lo, prm.box_hi)] * len(counts) if counts else None
    with pbf.Simulator(pos, vel, prm, counts=counts, boxes=boxes) as sim:
        sim.set_profiling(profiled)
        sim.time_step(0.0, steps)
        st = sim.stats()
        off, ids = sim.neighbors()
        pred = sim.predicted() if prm.flags & PBF_FLAG_KEEP_PREDICTED else np.zeros(0)
        return [sim.positions(), sim.velocities(), sim.densities(), off, ids, pred,
                np.array([st["mean_density"], st["mean_density_iter0"], st["max_density_error"], st["mean_neighbors"]])]


def _same(pos, vel, prm, **kw):
    for a, b in zip(_run(pos, vel, prm, False, **kw), _run(pos, vel, prm, True, **kw)):
        np.testing.assert_array_equal(a, b)


# a cluster up to 1,024 particles, 8 lanes a particle up to 2 x 152 blocks of 32, one lane up to 152
# blocks of 128 and of 256, above them the per-phase kernels
@pytest.mark.parametrize("n", [1, 31, 33, 64, 65, 500, 1024, 1025, 9727, 9729, 19455, 19457, 38911, 38913])
def test_same_bits_at_the_ends_of_the_forms(n):
    pos, vel, h = _state(n, seed=n)
    _same(pos, vel, scenes.physical_params(h, h / 2, flags=PBF_FLAG_STATS, max_neighbors=256))


@pytest.mark.parametrize("n", [700, 12000])
@pytest.mark.parametrize("iters,scorr_n", [(0, 4), (1, 4), (3, 3), (4, 6)])
def test_same_bits_for_iterations_and_exponents(n, iters, scorr_n):
    pos, vel, h = _state(n)
    flags = PBF_FLAG_GRAPH | PBF_FLAG_KEEP_PREDICTED
    _same(pos, vel, scenes.physical_params(h, h / 2, iters=iters, scorr_n=scorr_n, flags=flags, max_neighbors=256), steps=3)


@pytest.mark.parametrize("n", [150, 900])
def test_same_bits_with_long_lists_and_full_cells(n):  # over 64 entries, cells over 32 particles
    rng = np.random.default_rng(n)
    pos = 0.4 + 2.2 * H * rng.uniform(0, 1, (n, 3))
    prm = scenes.physical_params(H, H / 2, flags=PBF_FLAG_STATS, max_neighbors=1024)
    _same(pos, np.zeros_like(pos), prm, steps=1)


def test_same_bits_for_a_batch_and_a_fine_grid():
    counts = [1, 0, 40, 7, 1500, 33, 300]
    rng = np.random.default_rng(1)
    pos = np.concatenate([0.3 + 0.3 * rng.uniform(0, 1, (c, 3)) for c in counts])
    vel = rng.uniform(-1, 1, pos.shape)
    _same(pos, vel, scenes.physical_params(H, H / 2, flags=0, max_neighbors=1024), counts=counts)
    h = 0.021  # 125,000 cells: the tiles' sums are exchanged between blocks
    p = scenes.lattice(9, 9, 9, h / 2, corner=(0.1, 0.2, 0.3))
    _same(p, np.zeros_like(p), scenes.physical_params(h, h / 2, flags=0))


def test_alternating_with_the_per_phase_kernels():
    pos, vel, h = _state(3000)
    prm = scenes.physical_params(h, h / 2, flags=0, max_neighbors=256)
    with pbf.Simulator(pos, vel, prm) as a, pbf.Simulator(pos, vel, prm) as b:
        for k in range(6):
            a.set_profiling(k % 2 == 1)
            a.time_step(0.0, 1)
            if k == 3:
                assert np.array_equal(a.estimate_densities(), (b.time_step(0.0, 4), b.estimate_densities())[1])
        b.time_step(0.0, 2)
        np.testing.assert_array_equal(a.positions(), b.positions())
        np.testing.assert_array_equal(a.velocities(), b.velocities())
