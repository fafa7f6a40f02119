"""The per-phase neighbour build where a group's candidate window exceeds its tables and is read in
pieces, and where slots lie far apart along a row: the lists are those of the host's FP32 predicate,
and a clump costs no more a candidate than fluid near rest."""
import numpy as np
import pytest

from fluid_gb300 import pbf, scenes
from fluid_gb300.params import PBF_FLAG_KEEP_PREDICTED
from tests.helpers import csr_sets, neighbor_sets_fp32

pytestmark = pytest.mark.gpu

H = 0.05


def _lists(pos, **kw):
    prm = scenes.physical_params(H, H / 2, gravity=(0.0, 0.0, 0.0), flags=PBF_FLAG_KEEP_PREDICTED, **kw)
    with pbf.Simulator(pos, np.zeros_like(pos), prm) as sim:
        sim.set_profiling(True)  # a launch per phase also for few particles
        try:
            sim.time_step(0.0, 1)
        except pbf.PbfError as e:
            assert e.status == 5 and "neighbours" in str(e)
        return sim.predicted(), *sim.neighbors(), prm


# windows around one and two pieces of 448 candidates, several pieces, remainders of 32 and 8
@pytest.mark.parametrize("n", [440, 448, 449, 481, 500, 897, 900, 1000, 1500])
@pytest.mark.parametrize("extent", [0.04, 0.06])
def test_pieces(n, extent):
    rng = np.random.default_rng(n)
    far = rng.uniform(0.02, 0.3, (150, 3))
    pos = np.concatenate([0.45 + extent * rng.uniform(0, 1, (n, 3)), far])
    if extent == 0.04:  # every pair of a clump of at most 1,024 entries a list
        pos = pos[-(min(n, 1000) + 150):]
    xs, off, ids, prm = _lists(pos, max_neighbors=1024)
    want = csr_sets(*neighbor_sets_fp32(xs, prm.h2))
    got = csr_sets(off, ids)
    if max(map(len, want)) <= 1024:
        assert got == want
    else:  # full lists hold neighbours only
        assert all(g == w if len(w) <= 1024 else (len(g) == 1024 and g <= w) for g, w in zip(got, want))


@pytest.mark.parametrize("cap", [64, 200, 446, 448, 450, 600])
def test_capacity_inside_a_piece(cap):
    pos = 0.45 + 0.045 * np.random.default_rng(1).uniform(0, 1, (700, 3))
    xs, off, ids, prm = _lists(pos, max_neighbors=cap)
    want = csr_sets(*neighbor_sets_fp32(xs, prm.h2))
    assert max(map(len, want)) > cap
    for g, w in zip(csr_sets(off, ids), want):
        assert len(g) == min(len(w), cap) and g <= w


@pytest.mark.parametrize("n,rows", [(100, 1), (64, 2), (300, 1), (40000, 400)])
def test_slots_far_apart_along_rows(n, rows):
    rng = np.random.default_rng(n)
    x = rng.uniform(0.01, 0.99, n)
    r = rng.integers(0, rows, n)
    pos = np.stack([x, 0.03 + 0.045 * (r % 20), 0.03 + 0.045 * (r // 20)], 1) + rng.uniform(-0.01, 0.01, (n, 3))
    xs, off, ids, prm = _lists(pos, max_neighbors=256)
    assert csr_sets(off, ids) == csr_sets(*neighbor_sets_fp32(xs, prm.h2))


def test_a_clump_costs_no_more_a_candidate():
    h, us = 0.025, {}
    for r in (2.5, 3.0):  # 62 and 114 neighbours, windows of about 350 and 560 candidates
        pos = scenes.lattice(64, 64, 64, h / r, corner=(0.05,) * 3)
        pos = pos + np.random.default_rng(0).uniform(-0.05, 0.05, pos.shape) * h / r
        prm = scenes.physical_params(h, h / r, gravity=(0.0, 0.0, 0.0), iters=0, max_neighbors=256, flags=0)
        with pbf.Simulator(pos, np.zeros_like(pos), prm) as sim:
            sim.set_profiling(True)
            sim.time_step(1e-9, 5)
            best = np.inf
            for _ in range(5):
                sim.reset_phase_times()
                sim.time_step(1e-9, 5)
                best = min(best, sim.phase_times()["neighbors"][0])
            us[r] = best
    assert us[3.0] < 3.2 * us[2.5]  # 1.6 times the candidates, 1.8 times the entries
