"""Handles of small scenes that step at the same time, from two threads and from one, each step one
cooperative launch or one cluster: the states are those of each handle alone."""
import threading

import numpy as np
import pytest

from fluid_gb300 import pbf, scenes
from fluid_gb300.params import PBF_FLAG_GRAPH

pytestmark = pytest.mark.gpu

STEPS = 60


def _sim(n, flags):
    side = int(np.ceil(n ** (1 / 3)))
    s = 0.9 / max(side, 18)
    p = scenes.lattice(side, side, side, s, corner=(0.02, 0.0, 0.03))[:n]
    v = np.random.default_rng(n).uniform(-0.5, 0.5, p.shape)
    return pbf.Simulator(p, v, scenes.physical_params(2 * s, s, flags=flags, gravity=(0.0, 0.0, 0.0), max_neighbors=512))


def _alone(n, flags):
    with _sim(n, flags) as sim:
        assert sim.step_form > 0
        sim.time_step(1e-3, STEPS)
        return sim.positions(), sim.velocities()


@pytest.mark.parametrize("a,b", [(5000, 5000), (9000, 30000), (700, 15000), (38000, 38000)])
@pytest.mark.parametrize("flags", [0, PBF_FLAG_GRAPH])
def test_two_threads(a, b, flags):
    want = {n: _alone(n, flags) for n in {a, b}}
    got, errors = [None, None], []

    def work(k, n):
        try:
            with _sim(n, flags) as sim:
                for _ in range(STEPS // 10):
                    sim.time_step(1e-3, 10)
                got[k] = sim.positions(), sim.velocities()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k, n)) for k, n in enumerate((a, b))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for g, n in zip(got, (a, b)):
        np.testing.assert_array_equal(g[0], want[n][0])
        np.testing.assert_array_equal(g[1], want[n][1])


def test_two_streams_of_one_thread():
    sizes = (700, 5000, 9000, 30000)
    want = {n: _alone(n, 0) for n in sizes}
    sims = [_sim(n, 0) for n in sizes]
    for _ in range(STEPS):
        for sim in sims:
            sim.step_async(1e-3, 1)
    for sim, n in zip(sims, sizes):
        sim.sync()
        np.testing.assert_array_equal(sim.positions(), want[n][0])
        np.testing.assert_array_equal(sim.velocities(), want[n][1])
        sim.close()
