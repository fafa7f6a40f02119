"""A squared radius beyond FP32's range is infinity on the device: every particle of the scene is a
neighbour of every other one, and nothing else is, also where a turn of the warp scan is not full."""
import numpy as np
import pytest

from fluid_gb300 import pbf
from fluid_gb300.params import PbfParams
from tests.helpers import csr_sets

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("profiled", [False, True])  # the whole-step kernel, the per-phase kernels
@pytest.mark.parametrize("n", [1, 2, 31, 33, 40, 95, 300])
def test_all_pairs(n, profiled):
    prm = PbfParams(h=1e20, h2=1e40, iters=0, gravity=(0.0, 0.0, 0.0), box_lo=(0.0, 0.0, 0.0),
                    box_hi=(1.0, 1.0, 1.0), max_neighbors=512, flags=0)
    pos = np.random.default_rng(n).uniform(0.1, 0.9, (n, 3))
    with pbf.Simulator(pos, np.zeros_like(pos), prm) as sim:
        sim.set_profiling(profiled)
        try:
            sim.time_step(0.0, 1)
        except pbf.PbfError as e:  # infinite kernel values: PBF_ERR_NONFINITE, the lists are whole
            assert e.status == 4
        assert csr_sets(*sim.neighbors()) == [set(range(n)) - {i} for i in range(n)]
