"""The neighbour build's warp scan and its thread scan: neighbour sets against the host's FP32
predicate where groups, warps and tables end (partial warps, rows shared by few slots, several
scenes in a warp, candidate windows beyond the shared tables, pairs at exactly h)."""
import numpy as np
import pytest

from fluid_gb300 import pbf, scenes
from fluid_gb300.params import PBF_FLAG_KEEP_PREDICTED
from tests.helpers import csr_sets, neighbor_sets_fp32

pytestmark = pytest.mark.gpu

H = 0.05


def _params(**kw):
    return scenes.physical_params(H, H / 2, gravity=(0.0, 0.0, 0.0), flags=PBF_FLAG_KEEP_PREDICTED,
                                  max_neighbors=1024, **kw)


def _check(pos, counts=None):
    prm = _params()
    n = len(pos)
    boxes = [(prm.box_lo, prm.box_hi)] * len(counts) if counts else None
    with pbf.Simulator(pos, np.zeros_like(pos), prm, counts=counts, boxes=boxes) as sim:
        sim.time_step(0.0, 1)
        xs = sim.predicted()
        off, ids = sim.neighbors()
        assert sim.stats()["error_flags"] == 0
    got = csr_sets(off, ids)
    first = 0
    for c in counts or [n]:
        if c:
            want = csr_sets(*neighbor_sets_fp32(xs[first:first + c], prm.h2))
            assert [{j - first for j in s} for s in got[first:first + c]] == want
        first += c
    return max(len(s) for s in got) if got else 0


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 63, 65, 127, 129, 1000])
def test_partial_warps_and_rows(n):
    rng = np.random.default_rng(n)
    side = int(np.ceil(n ** (1 / 3)))
    p = scenes.lattice(side, side, side, H / 2, corner=(0.4, 0.4, 0.4))[:n]
    _check(p + rng.uniform(-0.2, 0.2, p.shape) * H / 2)


@pytest.mark.parametrize("n", [40, 600])
def test_one_row_of_cells(n):
    rng = np.random.default_rng(n)
    p = np.stack([rng.uniform(0.1, 0.9, n), np.full(n, 0.51), np.full(n, 0.52)], 1)
    _check(p + rng.uniform(-0.01, 0.01, p.shape) * [1, 1, 1])


@pytest.mark.parametrize("n", [50, 700, 5000])
def test_slots_scattered_over_rows(n):  # many groups to a warp, then few
    _check(np.random.default_rng(n).uniform(0.02, 0.98, (n, 3)))


@pytest.mark.parametrize("n,extent", [(300, 0.1), (700, 0.11), (900, 0.13)])
def test_windows_beyond_the_tables(n, extent):  # a dense clump: up to several hundred candidates a group
    rng = np.random.default_rng(n)
    p = 0.45 + extent * rng.uniform(0, 1, (n, 3))
    far = rng.uniform(0.02, 0.3, (200, 3))
    assert _check(np.concatenate([p, far])) > 40


def test_pairs_at_exactly_h():  # a lattice of spacing h / 2 in exact binary coordinates
    h = 0.0625
    p = scenes.lattice(9, 8, 7, h / 2, corner=(0.25, 0.25, 0.25))
    prm = scenes.physical_params(h, h / 2, gravity=(0.0, 0.0, 0.0), flags=PBF_FLAG_KEEP_PREDICTED)
    with pbf.Simulator(p, np.zeros_like(p), prm) as sim:
        sim.time_step(0.0, 1)
        xs = sim.predicted()
        off, ids = sim.neighbors()
    assert csr_sets(off, ids) == csr_sets(*neighbor_sets_fp32(xs, prm.h2))
    assert np.diff(off).max() == 32  # 26 around and 6 at exactly h


def test_several_scenes_in_a_warp():
    counts = [1, 3, 0, 8, 5, 40, 2, 17, 100, 9]
    rng = np.random.default_rng(0)
    p = np.concatenate([0.4 + 0.15 * rng.uniform(0, 1, (c, 3)) for c in counts])
    _check(p, counts)
