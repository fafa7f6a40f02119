"""The surface in two parts (pbf_surface_begin, pbf_surface_end) and Simulator.surface over them: room
for exactly the triangles, whatever their number, and the refusals of pbf_surface."""
import ctypes

import numpy as np
import pytest

from fluid_gb300 import pbf, scenes

pytestmark = pytest.mark.gpu

H = 0.05
BOX = dict(lo=(0.0, 0.0, 0.0), hi=(1.0, 1.0, 1.0))


def _sim(n=4000):
    prm = scenes.physical_params(H, H / 2, max_neighbors=256)
    pos = np.random.default_rng(n).uniform(0.05, 0.95, (n, 3))
    return pbf.Simulator(pos, np.zeros_like(pos), prm)


def _begin(sim, iso, step):
    count = ctypes.c_size_t(0)
    lo, hi = (np.array(BOX[k], dtype=np.float64) for k in ("lo", "hi"))
    sim._check(pbf.lib().pbf_surface_begin(sim._h, iso, step, pbf._ptr(lo), pbf._ptr(hi), ctypes.byref(count)))
    return count.value


def _end(sim, cap):
    xyz = np.full((cap, 3, 3), 7.0, dtype=np.float32)
    nrm = np.full((cap, 3, 3), 7.0, dtype=np.float32)
    sim._check(pbf.lib().pbf_surface_end(sim._h, pbf._ptr(xyz), pbf._ptr(nrm), cap))
    return xyz, nrm


def test_parts_and_whole():
    with _sim() as sim:
        iso = 0.05 * sim.params.rest_density
        xyz, nrm = sim.surface(iso=iso, step=0.3 * H, **BOX)
        t = len(xyz)
        assert t > 100000  # a blob of its own around most particles
        assert xyz.base is None and nrm.base is None and xyz.nbytes == 36 * t
        assert _begin(sim, iso, 0.3 * H) == t
        x, n = _end(sim, t + 5)
        assert np.array_equal(x[:t], xyz) and np.array_equal(n[:t], nrm) and (x[t:] == 7.0).all()
        _begin(sim, iso, 0.3 * H)
        x, n = _end(sim, 17)
        assert np.array_equal(x, xyz[:17]) and np.array_equal(n, nrm[:17])
        empty, _ = sim.surface(iso=1e30, **BOX)
        assert empty.shape == (0, 3, 3)


@pytest.mark.parametrize("step", [0.0, -1.0, 1e-160, 1e-320, 1e-6, float("nan"), float("inf")])
def test_steps_that_are_refused(step):
    with _sim(100) as sim:
        with pytest.raises(pbf.PbfError) as e:
            sim.surface(step=step, **BOX)
        assert e.value.status == 1


def test_an_end_without_its_beginning():
    with _sim() as sim:
        iso = 0.05 * sim.params.rest_density
        calls = {
            "twice": lambda: _end(sim, 10), "step": lambda: sim.time_step(1e-4, 1), "sort": sim.sort,
            "state": lambda: sim.set_state(sim.positions(), None), "at": lambda: sim.estimate_density_at(np.zeros((3, 3))),
            "restore": lambda: (sim.snapshot(), sim.restore()), "densities": sim.estimate_densities,
        }
        with pytest.raises(pbf.PbfError):
            _end(sim, 10)
        for call in calls.values():
            _begin(sim, iso, H)
            call()
            with pytest.raises(pbf.PbfError) as e:
                _end(sim, 10)
            assert e.value.status == 1
        _begin(sim, iso, H)
        sim.positions()  # a download leaves it open
        sim.stats()
        _end(sim, 10)
