"""A wait inside a small scene's step that gives up (a limit of one read): the launches behind it
return, every later call on the handle reports PBF_ERR_TIMEOUT, and other handles are unaffected."""
import numpy as np
import pytest

from fluid_gb300 import pbf, scenes
from fluid_gb300.params import PBF_FLAG_GRAPH, PBF_FLAG_KEEP_PREDICTED, PBF_FLAG_STATS

pytestmark = pytest.mark.gpu

TIMEOUT = 3  # PBF_ERR_TIMEOUT
H = 0.04


def _sim(n, flags, h=H):
    side = int(np.ceil(n ** (1 / 3)))
    s = min(h / 2, 0.9 / side)
    p = scenes.lattice(side, side, side, s, corner=(0.02, 0.0, 0.03))[:n]
    v = np.random.default_rng(n).uniform(-1, 1, p.shape)
    return pbf.Simulator(p, v, scenes.physical_params(2 * s, s, flags=flags))


def _refused(call, *args, **kw):
    with pytest.raises(pbf.PbfError) as e:
        call(*args, **kw)
    assert e.value.status == TIMEOUT


# 8 lanes a particle, one lane with blocks of 128 and of 256 threads
@pytest.mark.parametrize("n", [1025, 4096, 9000, 15000, 30000])
@pytest.mark.parametrize("flags", [0, PBF_FLAG_GRAPH | PBF_FLAG_STATS | PBF_FLAG_KEEP_PREDICTED])
def test_a_wait_that_gives_up(n, flags):
    with _sim(n, flags) as sim, _sim(n, flags) as other:
        sim.set_wait_limit(1)
        sim.step_async(0.0, 1)
        sim.set_wait_limit(0)
        sim.step_async(0.0, 3)  # in the stream before the host knows
        other.time_step(0.0, 2)
        _refused(sim.sync)
        for call in (sim.sync, sim.time_step, sim.step_async, sim.positions, sim.velocities, sim.densities,
                     sim.estimate_densities, sim.surface, sim.sort, sim.neighbors, sim.autotune):
            _refused(call)
        _refused(sim.estimate_density_at, np.zeros((1, 3)))
        assert sim.stats()["error_flags"] & 8
        sim.set_state(np.full((n, 3), 0.5), np.zeros((n, 3)))
        _refused(sim.time_step)
        with _sim(n, flags) as fresh:
            fresh.time_step(0.0, 2)
            np.testing.assert_array_equal(fresh.positions(), other.positions())
            np.testing.assert_array_equal(fresh.velocities(), other.velocities())


@pytest.mark.parametrize("first", ["profiled", "sort", "neighbors", "stats", "adjoint"])
def test_other_calls_before_the_host_knows(first):
    import torch
    n = 4096
    with _sim(n, 0) as sim:
        sim.set_wait_limit(1)
        sim.step_async(0.0, 1)
        if first == "profiled":  # the per-phase kernels, on cell counts that the step left
            sim.set_profiling(True)
            sim.step_async(0.0, 2)
        elif first == "sort":
            sim.sort()
        elif first == "neighbors":
            _refused(sim.neighbors)
        elif first == "stats":
            assert sim.stats()["error_flags"] & 8
        else:
            x = torch.rand((n, 3), device="cuda")
            g = [torch.zeros((n, 3), device="cuda") for _ in range(4)]
            r = torch.zeros(1, dtype=torch.float64, device="cuda")
            for pos in (x.data_ptr(), None):
                sim.adjoint_step_device(1e-3, pos, None, g[0].data_ptr(), g[1].data_ptr(), g[2].data_ptr(),
                                        g[3].data_ptr(), r.data_ptr())
        _refused(sim.sync)
        _refused(sim.time_step)


def test_clusters_wait_without_a_limit():
    with _sim(1000, 0, h=0.1) as a, _sim(1000, 0, h=0.1) as b:  # a grid of few cells
        a.set_wait_limit(1)
        a.time_step(0.0, 3)
        b.time_step(0.0, 3)
        np.testing.assert_array_equal(a.positions(), b.positions())


def test_a_generous_limit_changes_nothing():
    with _sim(5000, PBF_FLAG_GRAPH) as a, _sim(5000, PBF_FLAG_GRAPH) as b:
        a.time_step(0.0, 1)
        a.set_wait_limit(1 << 24)
        a.time_step(0.0, 2)
        b.time_step(0.0, 3)
        np.testing.assert_array_equal(a.positions(), b.positions())
